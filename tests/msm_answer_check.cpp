// Host driver for tests/test_msm_answer.py: the library thread that answers
// the MSM's last step (zk_gpu_b200/csrc/msm_answer.hpp), with this program in
// the kernel's place.  Exits 0 if the case named by argv[1] holds.
#include <dlfcn.h>
#include <pthread.h>
#include <sched.h>
#include <time.h>

#include <cerrno>
#include <cstring>
#include <vector>

#include "../zk_gpu_b200/csrc/msm_answer.hpp"

static bool g_no_threads = false;
// takes the place of the C library's for the whole program
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
  if (g_no_threads) return EAGAIN;
  using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  static const Fn real = (Fn)dlsym(RTLD_NEXT, "pthread_create");
  return real(t, a, f, arg);
}

namespace {
using namespace zk;
namespace fq = zk::host::fq;

struct Use {
  Mail mail{};
  Watch w;
  uint64_t want[12];
  Use() { w.mail = &mail; }
  // the kernel's part: sums that depend on `seed`, then the flag
  void prepare(uint32_t seed) {
    w.seq++;
    w.windows = 2 + seed % 3;
    w.c = 4 + seed % 5;
  }
  void raise(uint32_t seed) {
    fq::E one = fq::one(), two = fq::add(one, one);
    fq::Xyzz g{one, two, one, one};  // the generator (1, 2)
    std::memset(mail.win, 0, sizeof(mail.win));
    for (uint32_t i = 0; i < w.windows; i++) {
      if ((seed + i) % 4 == 0) continue;  // an identity among them
      fq::Xyzz p = g;
      for (uint32_t k = 0; k < (seed + 7 * i) % 11; k++) fq::xyzz_dbl(p);
      const fq::E* co[4] = {&p.x, &p.y, &p.zz, &p.zzz};
      for (int k = 0; k < 4; k++) std::memcpy(mail.win + 16 * i + 4 * k, co[k]->v, 32);
    }
    fq::msm_combine_windows(mail.win, w.windows, w.c, want);
    __atomic_store_n(&mail.ready, w.seq, __ATOMIC_RELEASE);
  }
  bool answered(int ms) {
    for (int i = 0; i < ms * 10; i++) {
      if (__atomic_load_n(&mail.done, __ATOMIC_ACQUIRE) == w.seq) return std::memcmp(mail.out, want, 96) == 0;
      std::this_thread::sleep_for(std::chrono::microseconds(100));
    }
    return false;
  }
  bool released(int ms) {
    for (int i = 0; i < ms * 10 && w.watched.load(); i++) std::this_thread::sleep_for(std::chrono::microseconds(100));
    return !w.watched.load();
  }
};

bool once(Use& u, uint32_t seed) {
  u.prepare(seed);
  if (!Answerer::get().watch(&u.w)) return false;
  u.raise(seed);
  return u.answered(5000) && u.released(5000);
}
}  // namespace

int main(int, char** argv) {
  const char* what = argv[1];
  if (!std::strcmp(what, "no thread to be had")) {
    static Use u;
    u.prepare(1);
    g_no_threads = true;
    if (Answerer::get().watch(&u.w) || u.w.watched.load()) return 1;
    g_no_threads = false;
    return once(u, 2) ? 0 : 1;
  }
  if (!std::strcmp(what, "ready long after")) {  // beyond the time it polls without pause
    static Use u;
    u.prepare(3);
    if (!Answerer::get().watch(&u.w)) return 1;
    std::this_thread::sleep_for(std::chrono::milliseconds(60));
    if (!u.w.watched.load()) return 1;
    u.raise(3);
    return u.answered(5000) && u.released(5000) ? 0 : 1;
  }
  if (!std::strcmp(what, "kernel not launched")) {  // dropped, then used again
    static Use u;
    u.prepare(6);
    if (!Answerer::get().watch(&u.w)) return 1;
    Answerer::drop(&u.w);
    return u.released(5000) && u.mail.done == 0 && once(u, 7) ? 0 : 1;
  }
  if (!std::strcmp(what, "many at once")) {  // 64 slots over four threads, used again and again
    std::atomic<int> bad{0};
    std::vector<std::thread> ts;
    for (uint32_t t = 0; t < 4; t++)
      ts.emplace_back([&bad, t] {
        std::vector<Use>* us = new std::vector<Use>(16);
        for (uint32_t r = 0; r < 60; r++) {
          for (uint32_t k = 0; k < 16; k++) {
            Use& u = (*us)[k];
            u.prepare(t * 977 + r * 16 + k);
            if (!Answerer::get().watch(&u.w)) bad++;
          }
          for (uint32_t k = 16; k-- > 0;) (*us)[k].raise(t * 977 + r * 16 + k);
          for (Use& u : *us)
            if (!u.answered(5000) || !u.released(5000)) bad++;
        }
      });
    for (auto& t : ts) t.join();
    return bad ? 1 : 0;
  }
  if (!std::strcmp(what, "one core for both")) {  // a program at work leaves its core only to the answers
    cpu_set_t set;
    CPU_ZERO(&set);
    CPU_SET(sched_getcpu(), &set);
    if (sched_setaffinity(0, sizeof(set), &set)) return 1;
    auto seconds = [](clockid_t c) {
      timespec t;
      clock_gettime(c, &t);
      return (double)t.tv_sec + 1e-9 * (double)t.tv_nsec;
    };
    static Use u;
    double mine = 0, all = 0;
    for (uint32_t r = 0; r < 20; r++) {
      u.prepare(r);
      if (!Answerer::get().watch(&u.w)) return 1;
      const double t0 = seconds(CLOCK_THREAD_CPUTIME_ID), p0 = seconds(CLOCK_PROCESS_CPUTIME_ID);
      for (const double end = seconds(CLOCK_MONOTONIC) + 0.015; seconds(CLOCK_MONOTONIC) < end;) {
      }
      mine += seconds(CLOCK_THREAD_CPUTIME_ID) - t0;
      all += seconds(CLOCK_PROCESS_CPUTIME_ID) - p0;
      u.raise(r);
      if (!u.answered(5000) || !u.released(5000)) return 1;
    }
    return mine > 0.75 * all ? 0 : 1;
  }
  if (!std::strcmp(what, "exit while watched")) {  // the thread is stopped, nobody is asked afterwards
    static Use u, v;
    if (!once(u, 4)) return 1;
    v.prepare(5);
    return Answerer::get().watch(&v.w) ? 0 : 1;
  }
  return 2;
}
