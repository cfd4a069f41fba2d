// Device results into ordinary (pageable) host memory.
//
// The driver copies to pageable memory at about 2.4 GB/s.  OutCopy goes
// through page-locked memory instead, and touches the destination's pages while
// the GPU still works (a fresh 90 MB array has 22000 of them, 5 ms to fault one
// after the other).  Up to 4 MB come over in one copy, queued behind the
// solve (stage), and are copied on by the caller (a thread costs 60-110 us to
// start, hidden behind most solves, and 40 to wake and join); more is split
// over 4 to 8 threads that each own a slot and move their chunks from the
// device into it and on, so that bus and memory overlap.  An exec beyond its loop, one B200: a
// 224^3 field (90 MB) 4.2 ms, 16 fields of 960^2 (118 MB) 5.0, a 101 x 120 x 77
// field (7.5 MB) 0.9; with one copy into page-locked memory followed by one out
// of it into untouched pages 6.3, 10 and 1.2.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <condition_variable>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace ws {

// Page-locked buffers, kept between solves (of any solver, on any thread) up
// to kKeep bytes in all; trim() gives the idle ones back.
class HostPool {
 public:
  static constexpr size_t kKeep = 128u << 20;
  void* get(size_t bytes, size_t* got) {
    {
      std::lock_guard<std::mutex> lock(mu_);
      int best = -1;
      for (int i = 0; i < (int)free_.size(); ++i)
        if (free_[i].bytes >= bytes && (best < 0 || free_[i].bytes < free_[best].bytes)) best = i;
      if (best >= 0) {
        const Buf b = free_[best];
        free_.erase(free_.begin() + best);
        idle_ -= b.bytes;
        *got = b.bytes;
        return b.p;
      }
    }
    size_t n = 64 << 10;
    while (n < bytes) n *= 2;
    void* p = nullptr;
    if (cudaHostAlloc(&p, n, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    *got = n;
    return p;
  }
  void put(void* p, size_t bytes) {
    if (!p) return;
    {
      std::lock_guard<std::mutex> lock(mu_);
      if (idle_ + bytes <= kKeep) try {
          free_.push_back(Buf{p, bytes});
          idle_ += bytes;
          return;
        } catch (const std::exception&) {  // no memory to remember it by: given back below
        }
    }
    cudaFreeHost(p);
  }
  void trim() {
    std::lock_guard<std::mutex> lock(mu_);
    for (const Buf& b : free_) cudaFreeHost(b.p);
    free_.clear();
    idle_ = 0;
  }

 private:
  struct Buf {
    void* p;
    size_t bytes;
  };
  std::mutex mu_;
  std::vector<Buf> free_;
  size_t idle_ = 0;
};

inline HostPool& host_pool() {
  static HostPool* pool = new HostPool;  // outlives every solver and the runtime's own end
  return *pool;
}

// A buffer of the pool for the length of a scope (where no page-locked memory is
// to be had, ordinary memory: slower copies), and until the device is done with
// it: a scope may be left with copies into it still queued (an error
// return), and the pool's next taker must not get them.
struct HostLease {
  void* p = nullptr;
  size_t bytes = 0;
  explicit HostLease(size_t n) {
    p = host_pool().get(n, &bytes);
    pooled_ = p != nullptr;
    if (!pooled_) p = std::malloc(n);
  }
  HostLease(const HostLease&) = delete;
  HostLease& operator=(const HostLease&) = delete;
  ~HostLease() {
    // (after an error the device may still hold it: then it is not used again)
    if (busy_ && cudaStreamSynchronize(stream_) != cudaSuccess) return;
    if (pooled_)
      host_pool().put(p, bytes);
    else
      std::free(p);
  }
  void queued(cudaStream_t stream) {  // copies on `stream` may write to it
    stream_ = stream;
    busy_ = true;
  }
  void settled() { busy_ = false; }  // the caller has waited for them

 private:
  cudaStream_t stream_ = nullptr;
  bool busy_ = false, pooled_ = false;
};

// The first of `group`, half of it, .. 1 for which make() finds memory (with its
// error, if it is another); *e: the last one's.
template <class Make>
int fitting_group(int group, Make make, cudaError_t* e) {
  while ((*e = make(group)) == cudaErrorMemoryAllocation && group > 1) {
    cudaGetLastError();
    group = (group + 1) / 2;
  }
  return group;
}

class OutCopy {
 public:
  // The threads touch dst's pages from here to run().
  OutCopy(void* dst, size_t bytes, int device)
      : dst_((char*)dst), bytes_(bytes), device_(device), whole_(bytes <= kWhole),
        chunk_(whole_ ? std::max<size_t>(bytes, 1) : std::min(kChunk, (bytes / 4 + 4095) / 4096 * 4096)),
        workers_(workers_of(bytes, chunk_)), slots_(workers_ * chunk_) {
    if (!slots_.p) return;
    try {
      threads_.reserve(workers_);  // nothing below may throw once a thread runs
      for (int w = 1; w < workers_; ++w) threads_.emplace_back([this, w] { work(w); });
    } catch (const std::exception&) {  // no threads or no memory: the caller takes the chunks of the missing ones
    }
  }
  ~OutCopy() { finish(-1); }
  bool ok() const { return slots_.p != nullptr; }
  void touch() {  // the caller's own pages
    for (int w = 0; w < workers_; ++w)
      if (w == 0 || w > (int)threads_.size()) touch_of(w);
  }
  // Queues the copy of src behind the work on `stream` (up to 4 MB; may be
  // queued again); run() follows once the caller has waited for the stream.
  cudaError_t stage(const void* src, cudaStream_t stream) {
    src_ = (const char*)src;
    stream_ = stream;
    if (!whole_) return cudaSuccess;
    slots_.queued(stream);
    return cudaMemcpyAsync(slots_.p, src, bytes_, cudaMemcpyDeviceToHost, stream);
  }
  // The staged result into the destination; returns when it is there.
  cudaError_t run() {
    slots_.settled();
    {
      std::lock_guard<std::mutex> lock(mu_);
      go_ = 1;
    }
    cv_.notify_all();
    for (int w = 0; w < workers_; ++w)
      if (w == 0 || w > (int)threads_.size()) copy_of(w);
    finish(1);
    return (cudaError_t)err_;
  }

 private:
  static constexpr size_t kWhole = 4u << 20, kChunk = 4u << 20;
  static int workers_of(size_t bytes, size_t chunk) {
    const size_t n = (bytes + chunk - 1) / chunk, hw = std::max(1u, std::thread::hardware_concurrency());
    return (int)std::max<size_t>(1, std::min<size_t>(n, std::min<size_t>(8, hw)));
  }
  void finish(int go) {
    {
      std::lock_guard<std::mutex> lock(mu_);
      if (!go_) go_ = go;
    }
    cv_.notify_all();
    for (std::thread& t : threads_)
      if (t.joinable()) t.join();
  }
  void work(int w) {
    touch_of(w);
    {
      std::unique_lock<std::mutex> lock(mu_);
      cv_.wait(lock, [this] { return go_ != 0; });
      if (go_ < 0) return;
    }
    copy_of(w);
  }
  // a byte of every page, unchanged; only bytes of the worker's own chunks
  void touch_of(int w) {
    for (size_t c = (size_t)w * chunk_; c < bytes_; c += (size_t)workers_ * chunk_) {
      const size_t end = std::min(bytes_, c + chunk_);
      for (size_t i = c; i < end; i = ((uintptr_t)(dst_ + i) / 4096 + 1) * 4096 - (uintptr_t)dst_) {
        volatile char* p = dst_ + i;
        *p = *p;
      }
    }
  }
  void copy_of(int w) {
    if (whole_) {
      std::memcpy(dst_, slots_.p, bytes_);
      return;
    }
    cudaEvent_t ev = nullptr;
    cudaError_t e = cudaSetDevice(device_);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    char* const slot = (char*)slots_.p + (size_t)w * chunk_;
    for (size_t c = (size_t)w * chunk_; c < bytes_ && e == cudaSuccess; c += (size_t)workers_ * chunk_) {
      const size_t n = std::min(chunk_, bytes_ - c);
      e = cudaMemcpyAsync(slot, src_ + c, n, cudaMemcpyDeviceToHost, stream_);
      if (e == cudaSuccess) e = cudaEventRecord(ev, stream_);
      if (e == cudaSuccess) e = cudaEventSynchronize(ev);
      if (e == cudaSuccess) std::memcpy(dst_ + c, slot, n);
    }
    if (ev) cudaEventDestroy(ev);
    if (e != cudaSuccess) {
      std::lock_guard<std::mutex> lock(mu_);
      err_ = (int)e;
      slots_.queued(stream_);  // a chunk may still be under way
    }
  }

  char* dst_;
  size_t bytes_;
  int device_;
  bool whole_;
  size_t chunk_;
  int workers_;
  HostLease slots_;
  std::vector<std::thread> threads_;
  std::mutex mu_;
  std::condition_variable cv_;
  int go_ = 0;
  int err_ = 0;
  const char* src_ = nullptr;
  cudaStream_t stream_ = nullptr;
};

}  // namespace ws
