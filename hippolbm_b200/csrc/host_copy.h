// host_copy.h -- device memory to the caller's pageable arrays.
//
// cudaMemcpy into pageable memory moves 3 to 4 GB/s: the driver stages it on one thread, which also takes
// the page faults of a fresh array.  Here chunks go through a pinned double buffer at the speed of the
// link while a few threads move the chunk before into place (and fault its pages in).  The buffer is the
// process's, 16 MiB, made at the first large read-out and given back by release(); one read-out uses it
// at a time, another one meanwhile takes the plain copy, as do pinned destinations and small ones.
// Measured without and with it (three alternations): populations FP64 128^3 65 / 24 ms, FP32 181 x 150 x 170
// 159 / 45; a serving stream of ten requests that keeps its results 60.1 / 56.3 (medians).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace hlbm {

class HostCopy {
 public:
  // dst <- src (device), ordered on s; a plain asynchronous copy, or complete on return
  cudaError_t copy(void* dst, const void* src, size_t bytes, cudaStream_t s) {
    cudaPointerAttributes at{};
    const bool known = cudaPointerGetAttributes(&at, dst) == cudaSuccess;
    if (!known) cudaGetLastError();
    if (bytes < SMALL || (known && at.type != cudaMemoryTypeUnregistered)) return plain(dst, src, bytes, s);
    std::unique_lock<std::mutex> lock(mutex_, std::try_to_lock);
    if (!lock.owns_lock()) return plain(dst, src, bytes, s);
    if (!buffer_ && cudaHostAlloc(&buffer_, 2 * CHUNK, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      buffer_ = nullptr;
      return plain(dst, src, bytes, s);
    }
    return staged(static_cast<char*>(dst), static_cast<const char*>(src), bytes, s);
  }

  // `rows` runs of `bytes` each, `pitch` bytes apart on the device, side by side in dst
  cudaError_t copy_rows(void* dst, const void* src, size_t pitch, size_t bytes, int rows, cudaStream_t s) {
    if (bytes < SMALL) return cudaMemcpy2DAsync(dst, bytes, src, pitch, bytes, rows, cudaMemcpyDeviceToHost, s);
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < rows && e == cudaSuccess; i++)
      e = copy(static_cast<char*>(dst) + i * bytes, static_cast<const char*>(src) + i * pitch, bytes, s);
    return e;
  }

  void release() {
    std::lock_guard<std::mutex> lock(mutex_);
    if (buffer_) cudaFreeHost(buffer_);
    buffer_ = nullptr;
  }

 private:
  static constexpr size_t CHUNK = size_t(8) << 20, SMALL = size_t(4) << 20;
  std::mutex mutex_;
  void* buffer_ = nullptr;

  static cudaError_t plain(void* dst, const void* src, size_t bytes, cudaStream_t s) {
    return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s);
  }

  cudaError_t staged(char* dst, const char* src, size_t bytes, cudaStream_t s) {
    const size_t chunks = (bytes + CHUNK - 1) / CHUNK;
    std::unique_ptr<std::atomic<int>[]> done(new (std::nothrow) std::atomic<int>[chunks]);
    if (!done) return plain(dst, src, bytes, s);
    for (size_t k = 0; k < chunks; k++) done[k].store(0);
    std::atomic<size_t> ready{0};  // chunks that have reached the pinned buffer
    std::atomic<bool> stop{false};
    std::atomic<int> team{0};  // threads that run; fixed before the first chunk is ready
    const auto length = [&](size_t k) { return std::min(CHUNK, bytes - k * CHUNK); };
    const auto move = [&](size_t k, int t, int n) {  // thread t's share of chunk k
      const size_t len = length(k), part = (len + n - 1) / n, a = std::min(len, part * t), b = std::min(len, a + part);
      std::memcpy(dst + k * CHUNK + a, static_cast<char*>(buffer_) + (k & 1) * CHUNK + a, b - a);
    };
    const auto work = [&](int t) {
      for (size_t k = 0; k < chunks; k++) {
        while (ready.load(std::memory_order_acquire) <= k) {
          if (stop.load(std::memory_order_relaxed)) return;
          std::this_thread::yield();
        }
        move(k, t, team.load(std::memory_order_relaxed));
        done[k].fetch_add(1, std::memory_order_release);
      }
    };
    std::vector<std::thread> threads;
    const unsigned cores = std::thread::hardware_concurrency();
    try {
      threads.reserve(8);
      for (int t = 0; t < int(std::min(8u, std::max(1u, cores))); t++) threads.emplace_back(work, t);
    } catch (...) {  // fewer threads, or none, than asked for
    }
    const int n = int(threads.size());
    team.store(n, std::memory_order_relaxed);
    cudaError_t e = cudaSuccess;
    for (size_t k = 0; k < chunks && e == cudaSuccess; k++) {
      if (k >= 2)
        while (done[k - 2].load(std::memory_order_acquire) < n) std::this_thread::yield();
      e = cudaMemcpyAsync(static_cast<char*>(buffer_) + (k & 1) * CHUNK, src + k * CHUNK, length(k), cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      if (e == cudaSuccess) {
        ready.store(k + 1, std::memory_order_release);
        if (n == 0) move(k, 0, 1);
      }
    }
    if (e != cudaSuccess) stop.store(true);
    for (std::thread& t : threads) t.join();
    return e;
  }
};

}  // namespace hlbm
