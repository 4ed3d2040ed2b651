// vls_hostcopy.h -- copies between pageable host arrays and the device.
//
// A pageable copy runs at 5-18 GB/s: one driver thread moves the bytes
// through its own staging and, into a fresh array, takes every page fault.
// Here large pageable copies go through two page-locked chunks, filled or
// emptied by all host threads while the other chunk is on the bus (the
// download of 135 MB into a fresh array, 16 host threads: 29 -> 10 ms; of
// 68 MB 14 -> 4.5 ms).
#pragma once
#include <cuda_runtime.h>
#include <omp.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>

namespace vls {

// memcpy by all host threads, in pieces of many pages
inline void parallel_copy(void *dst, const void *src, size_t n) {
  const size_t piece = (size_t)256 << 10;
  const int64_t np = (int64_t)((n + piece - 1) / piece);
#pragma omp parallel for schedule(static) if (np > 1)
  for (int64_t k = 0; k < np; ++k) {
    const size_t o = (size_t)k * piece;
    std::memcpy((char *)dst + o, (const char *)src + o, std::min(piece, n - o));
  }
}

// Page-locked chunk pairs shared by the objects of the process: a pair is one
// copy's while that copy runs; at most KEEP pairs wait for the next one, and
// the last object frees them.
class ChunkPool {
 public:
  static constexpr size_t CHUNK = (size_t)4 << 20;
  static constexpr size_t KEEP = 2;
  struct Pair {
    void *p[2] = {nullptr, nullptr};
  };
  static ChunkPool &get() {
    // never destroyed: objects with static storage may still copy at exit
    static ChunkPool *pool = new ChunkPool;
    return *pool;
  }
  void user(int d) {
    std::lock_guard<std::mutex> lk(m_);
    users_ += d;
    if (users_ == 0) {
      while (nfree_) drop(free_[--nfree_]);
    }
  }
  // false where no memory can be page-locked (the copy then goes without)
  bool take(Pair &q) {
    {
      std::lock_guard<std::mutex> lk(m_);
      if (nfree_) {
        q = free_[--nfree_];
        return true;
      }
    }
    for (int k = 0; k < 2; ++k)
      if (cudaHostAlloc(&q.p[k], CHUNK, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        q.p[k] = nullptr;
        drop(q);
        return false;
      }
    return true;
  }
  void give(Pair &q) {
    std::lock_guard<std::mutex> lk(m_);
    if (nfree_ < KEEP)
      free_[nfree_++] = q;
    else
      drop(q);
  }

 private:
  static void drop(Pair &q) {
    for (void *&p : q.p) {
      if (p) cudaFreeHost(p);
      p = nullptr;
    }
  }
  std::mutex m_;
  Pair free_[KEEP];
  size_t nfree_ = 0;
  int users_ = 0;
};

// One object's copies (one at a time, like the object's other calls; objects
// may copy at the same time in their own threads).
class HostCopy {
 public:
  // Smaller copies go to the runtime as they are: below it the chunks' first
  // allocation (several ms) and the threads' wake-ups cost what they save.
  static constexpr size_t MIN_BYTES = (size_t)16 << 20;

  HostCopy() { ChunkPool::get().user(1); }
  ~HostCopy() { ChunkPool::get().user(-1); }
  HostCopy(const HostCopy &) = delete;
  HostCopy &operator=(const HostCopy &) = delete;

  cudaError_t download(void *host, const void *dev, size_t bytes, cudaStream_t st) {
    ChunkPool::Pair q;
    if (!staged(host, bytes) || !ChunkPool::get().take(q))
      return cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st);
    return run(q, bytes, st, [&](size_t o, size_t n, void *chunk, int phase) {
      if (phase == 0)
        return cudaMemcpyAsync(chunk, (const char *)dev + o, n, cudaMemcpyDeviceToHost, st);
      parallel_copy((char *)host + o, chunk, n);
      return cudaSuccess;
    }, false);
  }
  cudaError_t upload(void *dev, const void *host, size_t bytes, cudaStream_t st) {
    ChunkPool::Pair q;
    if (!staged(host, bytes) || !ChunkPool::get().take(q))
      return cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st);
    return run(q, bytes, st, [&](size_t o, size_t n, void *chunk, int phase) {
      if (phase == 0) {
        parallel_copy(chunk, (const char *)host + o, n);
        return cudaMemcpyAsync((char *)dev + o, chunk, n, cudaMemcpyHostToDevice, st);
      }
      return cudaSuccess;
    }, true);
  }

  // after the object's stream has been synchronised
  void release() {
    for (cudaEvent_t &e : ev_) {
      if (e) cudaEventDestroy(e);
      e = nullptr;
    }
  }

 private:
  static bool staged(const void *host, size_t bytes) {
    // with one thread the copy in and out of the chunks is all serial: slower
    // than the driver's own (a download of 135 MB into an array in use 14.5
    // against 7.8 ms; 7.7 and 4.0 with two and sixteen threads)
    if (bytes < MIN_BYTES || omp_get_max_threads() < 2 || omp_in_parallel()) return false;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    return a.type == cudaMemoryTypeUnregistered;  // page-locked memory goes directly
  }
  // chunk k: phase 0 queues its copy, phase 1 comes when that copy is done.
  // Two chunks alternate; both copies are done on return.
  template <typename F>
  cudaError_t run(ChunkPool::Pair &q, size_t bytes, cudaStream_t st, F &&f, bool up) {
    constexpr size_t C = ChunkPool::CHUNK;
    cudaError_t e = cudaSuccess;
    for (cudaEvent_t &ev : ev_)
      if (!ev && (e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming)) != cudaSuccess) {
        ev = nullptr;
        ChunkPool::get().give(q);
        return e;
      }
    const size_t n = (bytes + C - 1) / C;
    auto done = [&](size_t k) {
      cudaError_t r = cudaEventSynchronize(ev_[k & 1]);
      if (r == cudaSuccess) r = f(k * C, std::min(C, bytes - k * C), q.p[k & 1], 1);
      return r;
    };
    // a chunk is filled again once its copy two chunks ago is done: uploads
    // wait for it before the fill, downloads empty the other chunk meanwhile
    for (size_t k = 0; k < n && e == cudaSuccess; ++k) {
      if (up && k >= 2) e = done(k - 2);
      if (e == cudaSuccess) e = f(k * C, std::min(C, bytes - k * C), q.p[k & 1], 0);
      if (e == cudaSuccess) e = cudaEventRecord(ev_[k & 1], st);
      if (e == cudaSuccess && !up && k >= 1) e = done(k - 1);
    }
    if (e == cudaSuccess && up && n >= 2) e = done(n - 2);
    if (e == cudaSuccess) e = done(n - 1);
    if (e != cudaSuccess) cudaStreamSynchronize(st);  // no copy may still use the chunks
    ChunkPool::get().give(q);
    return e;
  }
  cudaEvent_t ev_[2] = {nullptr, nullptr};
};

}  // namespace vls
