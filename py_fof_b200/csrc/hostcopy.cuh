// Host-to-device copies of ordinary (pageable) memory by several threads.
//
// cudaMemcpyAsync stages pageable memory through the driver's own pinned
// buffers on the calling thread (about 11 GB/s here, a fifth of the host
// link), and the call returns only when that is done.  StagedCopy instead
// deals the segments of a call, in order, as chunks to worker threads; each
// copies a chunk into a pinned buffer of its own and issues the copy from
// there, so the link sees several memcpys at once and the calling thread goes
// on with the work that does not need the later segments.
//
// The threads live for one call; the pinned buffers belong to the context.
#pragma once

#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "common.cuh"

namespace pyfof {

// Pinned chunk buffers and the events of the copies that read them.
struct CopyRing {
  static constexpr size_t kChunk = (size_t)1 << 20;
  static constexpr int kWorkers = 6, kSlots = 2;  // two buffers per worker: 12 MB
  uint8_t *mem = nullptr;
  cudaEvent_t ev[kWorkers * kSlots] = {};
  // true when the buffers are there (allocated on first use)
  bool ready() {
    if (mem) return true;
    if (cudaHostAlloc(reinterpret_cast<void **>(&mem), kChunk * kWorkers * kSlots, cudaHostAllocPortable) !=
        cudaSuccess) {
      cudaGetLastError();
      mem = nullptr;
      return false;
    }
    for (auto &e : ev)
      if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        release();
        return false;
      }
    return true;
  }
  void release() {
    for (auto &e : ev) {
      if (e) cudaEventDestroy(e);
      e = nullptr;
    }
    if (mem) cudaFreeHost(mem);
    mem = nullptr;
  }
};

class StagedCopy {
 public:
  // Below this many bytes in all, starting threads costs more than it saves.
  static constexpr size_t kMinBytes = (size_t)12 << 20;

  // Whether `src` is ordinary host memory (a pinned source copies directly).
  static bool pageable(const void *src) {
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, src) != cudaSuccess) {
      cudaGetLastError();
      return true;
    }
    return at.type == cudaMemoryTypeUnregistered;
  }

  // Whether the worker threads can read `src`: not device memory, which the
  // runtime's own copy takes like any other.
  static bool readable(const void *src) {
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, src) != cudaSuccess) {
      cudaGetLastError();
      return true;
    }
    return at.type != cudaMemoryTypeDevice;
  }

  ~StagedCopy() { join(); }

  // Appends a segment; its copies are issued on stream s.  Returns its index.
  int add(void *dst, const void *src, size_t bytes, cudaStream_t s) {
    Segment g;
    g.dst = static_cast<uint8_t *>(dst);
    g.src = static_cast<const uint8_t *>(src);
    g.bytes = bytes;
    g.stream = s;
    g.first = chunks_;
    g.n = (bytes + CopyRing::kChunk - 1) / CopyRing::kChunk;
    chunks_ += g.n;
    seg_.push_back(g);
    left_.push_back(g.n);
    return (int)seg_.size() - 1;
  }

  // Starts the workers; false (nothing started) when there are none to be had.
  bool start(CopyRing &ring, int device) {
    const unsigned hw = std::thread::hardware_concurrency();
    const int n = (int)std::min<size_t>(std::min<size_t>(CopyRing::kWorkers, hw / 2), chunks_);
    if (n < 2 || !ring.ready()) return false;
    device_ = device;
    try {
      for (int w = 0; w < n; ++w) threads_.emplace_back([this, &ring, w] { work(ring, w); });
    } catch (...) {  // no more threads: those that run take all chunks
      if (threads_.empty()) return false;
    }
    return true;
  }

  // Blocks until every copy of segment i has been issued on its stream.
  void wait(int i) {
    std::unique_lock<std::mutex> lk(mu_);
    cv_.wait(lk, [&] { return left_[i] == 0; });
  }

  // Ends the workers (all copies issued).  Returns the first CUDA error.
  cudaError_t join() {
    for (auto &t : threads_) t.join();
    threads_.clear();
    return error_;
  }

 private:
  struct Segment {
    uint8_t *dst;
    const uint8_t *src;
    size_t bytes, first, n;
    cudaStream_t stream;
  };

  void work(CopyRing &ring, int w) {
    cudaError_t e = cudaSetDevice(device_);
    bool used[CopyRing::kSlots] = {};
    for (int k = 0;; ++k) {
      const size_t c = next_.fetch_add(1);
      if (c >= chunks_) break;
      size_t i = 0;
      while (c >= seg_[i].first + seg_[i].n) ++i;
      const Segment &g = seg_[i];
      const size_t off = (c - g.first) * CopyRing::kChunk;
      const size_t len = std::min(CopyRing::kChunk, g.bytes - off);
      const int slot = k % CopyRing::kSlots, id = w * CopyRing::kSlots + slot;
      uint8_t *buf = ring.mem + (size_t)id * CopyRing::kChunk;
      if (e == cudaSuccess && used[slot]) e = cudaEventSynchronize(ring.ev[id]);
      if (e == cudaSuccess) {
        std::memcpy(buf, g.src + off, len);
        e = cudaMemcpyAsync(g.dst + off, buf, len, cudaMemcpyHostToDevice, g.stream);
      }
      if (e == cudaSuccess) e = cudaEventRecord(ring.ev[id], g.stream);
      used[slot] = true;
      std::lock_guard<std::mutex> lk(mu_);
      if (e != cudaSuccess && error_ == cudaSuccess) error_ = e;
      if (--left_[i] == 0) cv_.notify_all();
    }
    // the buffers are free for the next call once their copies are done
    for (int s = 0; s < CopyRing::kSlots; ++s)
      if (used[s] && e == cudaSuccess) e = cudaEventSynchronize(ring.ev[w * CopyRing::kSlots + s]);
    if (e != cudaSuccess) {
      std::lock_guard<std::mutex> lk(mu_);
      if (error_ == cudaSuccess) error_ = e;
    }
  }

  std::vector<Segment> seg_;
  std::vector<size_t> left_;  // copies not issued yet, per segment
  size_t chunks_ = 0;
  std::atomic<size_t> next_{0};
  std::vector<std::thread> threads_;
  std::mutex mu_;
  std::condition_variable cv_;
  cudaError_t error_ = cudaSuccess;
  int device_ = 0;
};

}  // namespace pyfof
