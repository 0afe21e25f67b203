// Large device-to-host copies into pageable memory.
//
// The runtime's own copy moves such a result through its staging buffer with
// one thread: 15 to 20 GB/s into resident pages, 6 GB/s into fresh ones (page
// faults), against 55 GB/s of the link.  Here the calling thread keeps a
// page-locked ring of pieces filled, and other threads copy the pieces out (and
// take the page faults) side by side.  Those make no CUDA calls: a thread's first
// one takes longer than a field of 5 MB.
//
// The ring is the process's, bounded (HOSTCOPY_RING bytes), allocated by the
// first large copy and freed with the last handle.  One copy uses it at a time;
// a copy of another thread that finds it taken goes the runtime's way.
#pragma once

#include <cuda_runtime.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <functional>
#include <mutex>
#include <thread>

namespace lbm {

constexpr int HOSTCOPY_THREADS = 8, HOSTCOPY_SLOTS = 16;
constexpr size_t HOSTCOPY_PIECE = 512 << 10;
constexpr size_t HOSTCOPY_RING = HOSTCOPY_SLOTS * HOSTCOPY_PIECE;
// Below this the threads cost what they save where the pages are resident:
// five fields of 5 MB (ten phase-by-phase steps with them) 4.4 ms without and
// 5.3 with, five of 11.5 MB (40 streamed steps) 14.4 and 15.1; five of 67 MB
// (80 steps at 256^3) 101 and 95 ms, into fresh pages 168 and 107; a frame of
// 158 MB (16 steps at 448x400x440, BF16) 99 and 77.
constexpr size_t HOSTCOPY_MIN = 16 << 20;

inline int hostcopy_threads(size_t bytes) {
  static const int cores = (int)std::thread::hardware_concurrency();
  const size_t most = std::min<size_t>(bytes / (2 * HOSTCOPY_PIECE), HOSTCOPY_THREADS);
  return std::max(1, std::min((int)most, cores / 2));
}

// up to N threads, as many as can be started, joined at the end
struct HostThreads {
  std::thread t[HOSTCOPY_THREADS];
  int started = 0;
  template <class F>
  HostThreads(int n, F &f) {
    try {
      for (; started < n; started++) t[started] = std::thread(std::ref(f));
    } catch (...) {  // the threads there are do the work
    }
  }
  ~HostThreads() {
    for (int i = 0; i < started; i++) t[i].join();
  }
};
// f() on this thread and on up to n - 1 others
template <class F>
inline void hostcopy_run(int n, F &f) {
  HostThreads others(n - 1, f);
  f();
}

struct HostRing {
  std::mutex mu;
  std::atomic<int> handles{0};
  std::atomic<long long> copies{0};  // that went through the ring (lbm_test_ring_copies)
  char *buf = nullptr;
  cudaEvent_t ev[HOSTCOPY_SLOTS] = {};
  int device = -1;  // the events'

  // the ring and its events, for copies from this device (current)
  bool ready(int dev) {
    if (!buf && cudaHostAlloc((void **)&buf, HOSTCOPY_RING, cudaHostAllocPortable) != cudaSuccess) buf = nullptr;
    if (buf && device != dev) {
      drop_events();
      bool ok = true;
      for (cudaEvent_t &e : ev) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
      if (ok) device = dev;
      else drop_events();
    }
    if (buf && device == dev) return true;
    cudaGetLastError();
    return false;
  }
  void drop_events() {
    for (cudaEvent_t &e : ev)
      if (e) cudaEventDestroy(e), e = nullptr;
    device = -1;
  }
  void attach() { handles++; }
  void detach() {
    if (--handles > 0) return;
    std::lock_guard<std::mutex> lk(mu);
    if (handles > 0 || !buf) return;
    drop_events();
    if (cudaFreeHost(buf) != cudaSuccess) cudaGetLastError();
    buf = nullptr;
  }
};
inline HostRing &host_ring() {
  static HostRing *r = new HostRing;  // (handles may outlive static destructors)
  return *r;
}

// neither page-locked nor managed: the copy engine cannot write it
inline bool pageable(const void *p) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, p) == cudaSuccess) return at.type == cudaMemoryTypeUnregistered;
  cudaGetLastError();
  return false;
}

// bytes from device memory to dst, complete on return, after the work that
// stream st holds.  st's device is current.
inline cudaError_t copy_to_host(void *dst, const void *src, size_t bytes, int device, cudaStream_t st) {
  HostRing &r = host_ring();
  std::unique_lock<std::mutex> lk(r.mu, std::defer_lock);
  const int n = hostcopy_threads(bytes);
  bool ring = bytes >= HOSTCOPY_MIN && n > 1 && pageable(dst) && lk.try_lock();
  if (ring) ring = r.ready(device);
  auto runtime = [&]() {
    if (lk.owns_lock()) lk.unlock();
    const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
    return e != cudaSuccess ? e : cudaStreamSynchronize(st);
  };
  if (!ring) return runtime();
  cudaError_t e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return e;

  constexpr size_t S = HOSTCOPY_SLOTS;
  const size_t pieces = (bytes + HOSTCOPY_PIECE - 1) / HOSTCOPY_PIECE;
  std::atomic<size_t> next{0}, landed{0};  // pieces claimed, pieces in the ring
  std::atomic<size_t> out[S] = {};         // pieces copied out of each slot
  std::atomic<bool> stop{false};
  auto length = [&](size_t k) { return std::min(HOSTCOPY_PIECE, bytes - k * HOSTCOPY_PIECE); };
  size_t issued = 0;
  auto issue = [&]() {  // every piece whose slot is free
    while (e == cudaSuccess && issued < pieces && out[issued % S].load(std::memory_order_acquire) == issued / S) {
      const size_t k = issued;
      e = cudaMemcpyAsync(r.buf + k % S * HOSTCOPY_PIECE, (const char *)src + k * HOSTCOPY_PIECE, length(k),
                          cudaMemcpyDeviceToHost, st);
      if (e == cudaSuccess) e = cudaEventRecord(r.ev[k % S], st);
      if (e == cudaSuccess) issued++;
    }
  };
  auto work = [&]() {
    for (size_t k = next++; k < pieces; k = next++) {
      while (landed.load(std::memory_order_acquire) <= k) {
        if (stop.load(std::memory_order_relaxed)) return;
        std::this_thread::yield();
      }
      memcpy((char *)dst + k * HOSTCOPY_PIECE, r.buf + k % S * HOSTCOPY_PIECE, length(k));
      out[k % S].fetch_add(1, std::memory_order_release);
    }
  };
  issue();
  int started = 0;
  {
    HostThreads threads(n, work);
    started = threads.started;
    for (size_t k = 0; started && e == cudaSuccess && k < pieces;) {
      issue();
      if (e != cudaSuccess) break;
      if (issued == k) {
        std::this_thread::yield();
        continue;
      }
      e = cudaEventSynchronize(r.ev[k % S]);
      if (e == cudaSuccess) landed.store(++k, std::memory_order_release);
    }
    if (e != cudaSuccess) stop = true;
  }
  if (e != cudaSuccess || !started) {
    // copies into the ring may be in flight
    const cudaError_t e2 = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = e2;
    return e != cudaSuccess ? e : runtime();
  }
  r.copies++;
  return cudaSuccess;
}

}  // namespace lbm
