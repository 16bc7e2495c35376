// Device memory -> the caller's host buffer.
//
// A copy into pageable memory goes through the driver's staging
// buffers on one host thread, which also takes the page faults of a fresh
// array: 3 to 5 GB/s where the link carries 52. Such a copy is cut into parts,
// one host thread each, with two pinned buffers per thread: while one chunk
// arrives the thread copies the one before. (Six porous boxes in a batch,
// admission to read-back of 205 MB: 187 -> 152 ms.) Pinned destinations and
// copies below 4 MiB go directly.
//
// The objects of a process share the 8 MiB of pinned buffers and the streams.
// They take some milliseconds to make, so a copy of 16 MiB or more makes them
// first; they are given back with the last object. They serve one copy at a
// time, on the device they were made on; a copy that finds them taken goes
// directly.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace tclb {

class ReadBackPool {
 public:
  static ReadBackPool& get() {
    static ReadBackPool* p = new ReadBackPool;  // never destroyed: the CUDA runtime may be gone by then
    return *p;
  }
  void enter() {
    std::lock_guard<std::mutex> l(m_);
    users_++;
  }
  void leave() {
    std::lock_guard<std::mutex> l(m_);
    if (--users_ > 0) return;
    std::lock_guard<std::mutex> b(busy_);
    release();
  }
  // Copy `bytes` after the work enqueued on s; returns when dst holds them.
  cudaError_t copy(void* dst, const void* src, size_t bytes, cudaStream_t s, int device) {
    std::unique_lock<std::mutex> l(busy_, std::defer_lock);
    if (bytes < PARALLEL_BYTES || pinned(dst) || !l.try_lock() || (lanes_.empty() && bytes < FIRST_BYTES) ||
        !prepare(device)) {
      const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s);
      return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
    }
    cudaError_t e = cudaStreamSynchronize(s);  // the parts are copied on streams of their own
    if (e != cudaSuccess) return e;
    const size_t n = lanes_.size(), part = ((bytes + n - 1) / n + 4095) / 4096 * 4096;
    cudaError_t err[MAX_LANES] = {};
    std::vector<std::thread> threads;
    auto run = [&](size_t k, bool own) {  // own: in a thread of its own, whose current device is not set
      const size_t at = std::min(k * part, bytes), end = std::min(at + part, bytes);
      err[k] = copy_part(lanes_[k], static_cast<char*>(dst) + at, static_cast<const char*>(src) + at, end - at,
                         own ? device : -1);
    };
    size_t started = 1;
    try {
      threads.reserve(n);
      for (; started < n; started++) threads.emplace_back(run, started, true);
    } catch (const std::exception&) {  // no more threads: the rest runs here
    }
    run(0, false);
    for (size_t k = started; k < n; k++) run(k, false);
    for (auto& t : threads) t.join();
    for (cudaError_t x : err)
      if (x != cudaSuccess) return x;
    return cudaSuccess;
  }

 private:
  static constexpr size_t PARALLEL_BYTES = (size_t)4 << 20, FIRST_BYTES = (size_t)16 << 20, CHUNK = (size_t)512 << 10;
  static constexpr unsigned MAX_LANES = 8;
  struct Lane {
    char* buf[2] = {nullptr, nullptr};  // in buffers_
    cudaEvent_t event[2] = {nullptr, nullptr};
    cudaStream_t stream = nullptr;
  };
  std::mutex m_, busy_;  // the count of objects; the lanes
  int users_ = 0, device_ = -1;
  std::vector<Lane> lanes_;
  char* buffers_ = nullptr;

  static bool pinned(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    return a.type != cudaMemoryTypeUnregistered;
  }

  void release() {
    for (Lane& l : lanes_) {
      for (int b = 0; b < 2; b++)
        if (l.event[b]) cudaEventDestroy(l.event[b]);
      if (l.stream) cudaStreamDestroy(l.stream);
    }
    lanes_.clear();
    if (buffers_) cudaFreeHost(buffers_);
    buffers_ = nullptr;
  }

  bool prepare(int device) {
    if (!lanes_.empty()) return device == device_;
    const size_t n = std::max(1u, std::min(MAX_LANES, std::thread::hardware_concurrency() / 2));
    try {
      lanes_.resize(n);
    } catch (const std::exception&) {
      return false;
    }
    bool ok = cudaMallocHost(reinterpret_cast<void**>(&buffers_), n * 2 * CHUNK) == cudaSuccess;
    for (size_t k = 0; k < n && ok; k++) {
      Lane& l = lanes_[k];
      ok = cudaStreamCreateWithFlags(&l.stream, cudaStreamNonBlocking) == cudaSuccess;
      for (int b = 0; b < 2 && ok; b++) {
        l.buf[b] = buffers_ + (2 * k + b) * CHUNK;
        ok = cudaEventCreateWithFlags(&l.event[b], cudaEventDisableTiming) == cudaSuccess;
      }
    }
    if (!ok) {
      cudaGetLastError();
      release();
      return false;
    }
    device_ = device;
    return true;
  }

  static cudaError_t copy_part(Lane& l, char* dst, const char* src, size_t bytes, int device) {
    cudaError_t e = device >= 0 ? cudaSetDevice(device) : cudaSuccess;
    const size_t chunks = (bytes + CHUNK - 1) / CHUNK;
    auto fetch = [&](size_t i) {
      const size_t n = std::min(CHUNK, bytes - i * CHUNK);
      cudaError_t r = cudaMemcpyAsync(l.buf[i & 1], src + i * CHUNK, n, cudaMemcpyDeviceToHost, l.stream);
      return r == cudaSuccess ? cudaEventRecord(l.event[i & 1], l.stream) : r;
    };
    if (e == cudaSuccess && chunks > 0) e = fetch(0);
    for (size_t i = 0; i < chunks && e == cudaSuccess; i++) {
      if (i + 1 < chunks) e = fetch(i + 1);
      if (e == cudaSuccess) e = cudaEventSynchronize(l.event[i & 1]);
      if (e == cudaSuccess) std::memcpy(dst + i * CHUNK, l.buf[i & 1], std::min(CHUNK, bytes - i * CHUNK));
    }
    if (e != cudaSuccess) cudaStreamSynchronize(l.stream);  // nothing in flight into the buffers
    return e;
  }
};

// An object's share of the pool.
class ReadBack {
 public:
  ReadBack() { ReadBackPool::get().enter(); }
  ~ReadBack() { ReadBackPool::get().leave(); }
  ReadBack(const ReadBack&) = delete;
  ReadBack& operator=(const ReadBack&) = delete;
  cudaError_t copy(void* dst, const void* src, size_t bytes, cudaStream_t s, int device) {
    return ReadBackPool::get().copy(dst, src, bytes, s, device);
  }
};

}  // namespace tclb
