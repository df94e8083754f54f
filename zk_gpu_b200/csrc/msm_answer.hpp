// msm_answer.hpp — the host side of the MSM's last step (msm_combine.cu): the
// slots through which a stream's last kernel passes its window sums, and the
// library thread that answers them.  No CUDA here: the tests compile this file
// for the host alone and play the kernel's part.
#pragma once
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstdlib>
#include <mutex>
#include <thread>

#include "host_field.hpp"

namespace zk {

// pinned, read and written by both sides
struct Mail {
  uint32_t ready;  // the kernel's: sequence number of the sums in `win`
  uint32_t done;   // the host's: sequence number of the answer in `out`
  uint32_t pad[2];
  uint64_t win[MSM_MAX_WINDOWS * 16];
  uint64_t out[12];
};

// A slot's use as the library thread sees it; `next` and the values above it
// belong to the thread while `watched`.
struct Watch {
  Mail* mail = nullptr;
  uint32_t seq = 0, windows = 0, c = 0;
  Watch* next = nullptr;
  std::atomic<bool> watched{false};  // the library thread has not answered yet
  std::atomic<bool> dropped{false};  // its kernel will not come
};

// The thread that answers.  It polls while slots are watched, for 20 ms after
// the last event without pause but yielding its core, then with short sleeps,
// and sleeps otherwise.
class Answerer {
 public:
  static Answerer& get() {
    static Answerer* a = new Answerer();  // stopped at exit, never destroyed
    return *a;
  }
  // Answer w (not watched now) once its kernel is ready.  False, and nothing
  // started, if nobody will: at exit, or when the thread cannot be had.  Asked
  // before the kernel is launched: where launches wait for their kernels
  // (CUDA_LAUNCH_BLOCKING, a serialising profiler) nobody would answer it else.
  bool watch(Watch* w) {
    std::lock_guard<std::mutex> lk(mu_);
    if (stop_) return false;
    if (!thread_.joinable()) {
      try {
        thread_ = std::thread([this] { run(); });
      } catch (...) {  // the C entry that asks must not let this through
        return false;
      }
      // registered after the CUDA runtime's own handlers, so it runs before
      // they unmap the slots; kernels still waiting do the step themselves
      std::atexit([] { get().stop(); });
    }
    w->dropped.store(false);
    w->watched.store(true);
    w->next = queue_;
    queue_ = w;
    queued_.store(true);
    cv_.notify_one();
    return true;
  }
  // w's kernel was not launched after all; it stays watched until the thread
  // has let go of it.
  static void drop(Watch* w) { w->dropped.store(true); }

 private:
  void stop() {
    {
      std::lock_guard<std::mutex> lk(mu_);
      stop_ = true;
      queued_.store(true);
      cv_.notify_one();
    }
    if (thread_.joinable()) thread_.join();
  }
  void run() {
    using clk = std::chrono::steady_clock;
    Watch* watched = nullptr;
    clk::time_point last = clk::now();
    for (;;) {
      if (queued_.load() || !watched) {
        std::unique_lock<std::mutex> lk(mu_);
        cv_.wait(lk, [&] { return stop_ || queue_ || watched; });
        if (stop_) return;
        while (Watch* w = queue_) {
          queue_ = w->next;
          w->next = watched;
          watched = w;
        }
        queued_.store(false);
        last = clk::now();
      }
      for (Watch** at = &watched; *at;) {
        Watch* w = *at;
        if (__atomic_load_n(&w->mail->ready, __ATOMIC_ACQUIRE) == w->seq) {
          host::fq::msm_combine_windows(w->mail->win, w->windows, w->c, w->mail->out);
          __atomic_store_n(&w->mail->done, w->seq, __ATOMIC_RELEASE);
        } else if (!w->dropped.load()) {
          at = &w->next;
          continue;
        }
        *at = w->next;  // before the slot may be used again
        w->watched.store(false, std::memory_order_release);
        last = clk::now();
      }
      if (watched && clk::now() - last > std::chrono::milliseconds(20))
        std::this_thread::sleep_for(std::chrono::microseconds(20));
      else
        std::this_thread::yield();  // the core to whoever else wants it
    }
  }
  std::mutex mu_;
  std::condition_variable cv_;
  Watch* queue_ = nullptr;
  std::atomic<bool> queued_{false};
  bool stop_ = false;
  std::thread thread_;
};

}  // namespace zk
