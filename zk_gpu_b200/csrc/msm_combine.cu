// msm_combine.cu — the last step of a device-resident MSM: Horner over the
// window sums, sum_w 2^(c w) W_w, and the normalisation.
//
// The ~250 doublings of this step depend on one another: a GPU thread needs
// 1.3 ms for them, a host core 70 us.  A host function on the stream
// (cudaLaunchHostFunc) gives them to the host, but starts 50 us after the work
// before it when the caller waits and 170-420 us after it when the caller goes
// on enqueueing (measured on B200 hosts), which was half of a 2^14-point MSM.
// So the stream's last kernel hands the sums over itself: it writes them to a
// pinned slot, raises its flag and waits for the answer, which a library thread
// that watches the slots writes next to them.
//
// The wait is bounded (ZKGPU_MSM_HOST_WAIT_US, default 3000): when the host has
// not answered by then (it is stopped, or overcommitted), the kernel does the
// step by itself, as it does at once while the stream is being captured into a
// graph, whose replays have no slot.  Either way the result is the same.
//
// Slots are pooled per device, at most kMaxSlots; one is used again when its
// kernel has finished and the library thread is done with it.
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <vector>

#include "curve.cuh"
#include "fq_inv.cuh"
#include "msm.cuh"
#include "msm_answer.hpp"
#include "msm_field.cuh"
#include "runtime.cuh"

namespace zk {

namespace {

__device__ __forceinline__ uint32_t ld_acquire_sys(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_sys(uint32_t* p, uint32_t v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint64_t now_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// The caller's result is an array of 64-bit words: 8-byte stores.
__device__ __forceinline__ void st_words(uint64_t* out, const uint32_t r[8]) {
#pragma unroll
  for (int k = 0; k < 4; k++) out[k] = (uint64_t)r[2 * k + 1] << 32 | r[2 * k];
}

__device__ __noinline__ void combine_here(const fe* winsum, uint32_t windows, uint32_t c, uint64_t* out) {
  xyzz_t acc, w;
  ld_xyzz(acc, winsum + 4 * (uint64_t)(windows - 1));
#pragma unroll 1
  for (int i = (int)windows - 2; i >= 0; i--) {
#pragma unroll 1
    for (uint32_t k = 0; k < c; k++) xyzz_dbl(acc, acc);
    ld_xyzz(w, winsum + 4 * (uint64_t)i);
    xyzz_add(acc, w);
  }
  aff_t p;
  uint32_t z[8];
  set_zero(p.x);
  set_zero(p.y);
  set_zero(z);
  if (!xyzz_is_inf(acc)) {
    uint32_t t[8];
    qmul(t, acc.zz, acc.zzz);
    fq_inv_mont(t, t);
    qmul(z, t, acc.zzz);  // 1 / ZZ
    qmul(p.x, acc.x, z);
    qmul(z, t, acc.zz);   // 1 / ZZZ
    qmul(p.y, acc.y, z);
    reduce_once<P_q>(p.x, p.x);
    reduce_once<P_q>(p.y, p.y);
    set_one<P_q>(z);
  }
  st_words(out, p.x);
  st_words(out + 4, p.y);
  st_words(out + 8, z);
}

__global__ void __launch_bounds__(128) msm_combine_kernel(const fe* winsum, uint32_t windows, uint32_t c, uint64_t* out,
                                                          Mail* mail, uint32_t seq, uint64_t wait_ns) {
  if (mail) {
    __shared__ uint32_t answered;
    const uint4* src = reinterpret_cast<const uint4*>(winsum);
    uint4* dst = reinterpret_cast<uint4*>(mail->win);
    for (uint32_t i = threadIdx.x; i < windows * 8; i += blockDim.x) dst[i] = src[i];
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) {
      st_release_sys(&mail->ready, seq);
      const uint64_t t0 = now_ns();
      uint32_t got;
      while (!(got = ld_acquire_sys(&mail->done) == seq) && now_ns() - t0 < wait_ns) __nanosleep(100);
      answered = got;
    }
    __syncthreads();
    if (answered) {
      if (threadIdx.x < 12) out[threadIdx.x] = *(volatile const uint64_t*)&mail->out[threadIdx.x];
      return;
    }
  }
  if (threadIdx.x == 0) combine_here(winsum, windows, c, out);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
struct Slot : Watch {
  cudaEvent_t used = nullptr;  // its last kernel has finished
  bool taken = false;          // between acquire and the event record
};
constexpr size_t kMaxSlots = 64;

std::mutex g_slot_mu;
std::vector<std::vector<std::unique_ptr<Slot>>> g_slots;  // per device

// A free slot, made if there is none, or null when all kMaxSlots are in use, a
// new one cannot be had or an event cannot be asked (the caller's kernel then
// does the step itself); no error is left behind.
Slot* acquire_slot(int dev) try {
  std::lock_guard<std::mutex> lk(g_slot_mu);
  if ((int)g_slots.size() <= dev) g_slots.resize(dev + 1);
  auto& pool = g_slots[dev];
  for (auto& s : pool) {
    if (s->taken || s->watched.load(std::memory_order_acquire)) continue;
    const cudaError_t q = cudaEventQuery(s->used);
    if (q != cudaSuccess) cudaGetLastError();
    if (q == cudaErrorNotReady) continue;
    if (q != cudaSuccess) return nullptr;
    s->taken = true;
    return s.get();
  }
  if (pool.size() >= kMaxSlots) return nullptr;
  pool.reserve(kMaxSlots);
  auto s = std::make_unique<Slot>();
  if (cudaMallocHost((void**)&s->mail, sizeof(Mail)) != cudaSuccess ||
      cudaEventCreateWithFlags(&s->used, cudaEventDisableTiming) != cudaSuccess) {
    if (s->mail) cudaFreeHost(s->mail);
    cudaGetLastError();
    return nullptr;
  }
  std::memset(s->mail, 0, sizeof(Mail));
  s->taken = true;
  pool.push_back(std::move(s));
  return pool.back().get();
} catch (const std::bad_alloc&) {
  return nullptr;
}

void release_slot(Slot* s) {
  std::lock_guard<std::mutex> lk(g_slot_mu);
  s->taken = false;
}

uint64_t host_wait_ns() {
  static const uint64_t ns = [] {
    const char* v = std::getenv("ZKGPU_MSM_HOST_WAIT_US");
    return (v && *v ? std::strtoull(v, nullptr, 10) : 3000ull) * 1000ull;
  }();
  return ns;
}

}  // namespace

cudaError_t msm_combine(const fe* d_winsum, uint32_t windows, uint32_t c, uint64_t* d_out, cudaStream_t s) {
  if (windows == 0 || windows > MSM_MAX_WINDOWS) return cudaErrorInvalidValue;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  e = cudaStreamIsCapturing(s, &cap);
  if (e != cudaSuccess) return e;
  const uint64_t wait = host_wait_ns();
  Slot* slot = cap == cudaStreamCaptureStatusNone && wait ? acquire_slot(dev) : nullptr;
  if (slot) {
    slot->seq++;
    slot->windows = windows;
    slot->c = c;
    if (!Answerer::get().watch(slot)) {
      release_slot(slot);
      slot = nullptr;
    }
  }
  msm_combine_kernel<<<1, 128, 0, s>>>(d_winsum, windows, c, d_out, slot ? slot->mail : nullptr, slot ? slot->seq : 0,
                                       wait);
  e = cudaGetLastError();
  if (!slot) return e;
  if (e != cudaSuccess) {
    Answerer::drop(slot);
  } else {
    // without the event nobody can tell when the kernel is done with its slot:
    // it stays taken
    e = cudaEventRecord(slot->used, s);
    if (e != cudaSuccess) return e;
  }
  release_slot(slot);
  return e;
}

}  // namespace zk
