// Copies of a wave packet between pageable host memory (complex128) and the device (complex128 or complex64) by several
// host threads. One cudaMemcpyAsync of pageable memory runs at the speed of one core copying into the driver's staging
// buffer, plus, for a freshly allocated destination, one core's page faults (5 GB/s together for the restart of a
// 134 MB packet). Here every thread takes chunks in turn through two pinned buffers and a stream of its own, and the
// mixed form's conversion is done on the way, so that half the bytes cross the bus.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <thread>
#include <type_traits>
#include <vector>

namespace spo_host {

// The streams and pinned buffers of a device's large copies: at most 8 MiB of pinned memory, made for the first handle
// that needs them, shared by all handles of the device (one copy at a time) and freed with the last of them.
class CopyPool {
 public:
  static constexpr std::size_t kChunk = 512 << 10;  // bytes on the device per chunk
  struct Worker {
    cudaStream_t stream = nullptr;
    cudaEvent_t done[2] = {nullptr, nullptr};
    char* buffer[2] = {nullptr, nullptr};
  };
  std::mutex busy;
  std::vector<Worker> workers;

  // The pool of a device (the current one), made if `make` and there is none; null if there is none or it cannot be had.
  static std::shared_ptr<CopyPool> of_device(int device, bool make) {
    static std::mutex mutex;
    static std::map<int, std::weak_ptr<CopyPool>> pools;
    std::lock_guard<std::mutex> lock(mutex);
    std::shared_ptr<CopyPool> p = pools[device].lock();
    if (p || !make) return p;
    p = std::make_shared<CopyPool>();
    if (p->prepare() != cudaSuccess) {
      (void)cudaGetLastError();
      return nullptr;
    }
    pools[device] = p;
    return p;
  }
  ~CopyPool() {
    for (Worker& w : workers) {
      if (w.stream) cudaStreamDestroy(w.stream);
      for (cudaEvent_t d : w.done)
        if (d) cudaEventDestroy(d);
    }
    if (pinned_) cudaFreeHost(pinned_);
  }

 private:
  cudaError_t prepare() {
    const unsigned cores = std::thread::hardware_concurrency();
    workers.resize(std::max(1u, std::min(8u, cores / 2)));
    cudaError_t e = cudaMallocHost(reinterpret_cast<void**>(&pinned_), 2 * kChunk * workers.size());
    for (std::size_t k = 0; k < workers.size() && e == cudaSuccess; ++k) {
      Worker& w = workers[k];
      e = cudaStreamCreateWithFlags(&w.stream, cudaStreamNonBlocking);
      for (int b = 0; b < 2 && e == cudaSuccess; ++b) {
        e = cudaEventCreateWithFlags(&w.done[b], cudaEventDisableTiming);
        w.buffer[b] = pinned_ + (2 * k + b) * kChunk;
      }
    }
    return e;
  }
  char* pinned_ = nullptr;
};

// A handle's large copies. Not thread-safe, as the handle is not; several handles may copy from several threads.
class RawCopier {
 public:
  static constexpr std::size_t kChunk = CopyPool::kChunk;
  // Host bytes from which a copy is faster this way (18 MiB of a mixed packet up 1.2 -> 0.8 ms, down 1.1 -> 0.9; 9 MiB up 0.6
  // -> 0.5, down 0.6 -> 0.8).
  static constexpr std::size_t kMin = 16 << 20;
  // The pool costs 6 to 13 ms to make and 1 to 8 to give back; the copies gain about 0.2 ms per MiB. So a handle that finds
  // none uses plain copies for the first 64 MiB of those that would have taken this path: a program that reads one small
  // packet at its end does not pay for it (10 ms against 1), one that goes on has it after a few copies.
  static constexpr std::size_t kWorth = 64 << 20;
  using Worker = CopyPool::Worker;

  // Whether a copy of n host bytes from or to p takes this path: large, p not pinned (whose copies run at bus speed), and the
  // pool is there, or worth making and to be had. If not, the caller copies by cudaMemcpyAsync.
  bool wanted(const void* p, std::size_t n, int device) {
    if (n < kMin) return false;
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
      (void)cudaGetLastError();
      return false;
    }
    if (a.type != cudaMemoryTypeUnregistered) return false;
    if (pool_) return true;
    copied_ += n;
    pool_ = CopyPool::of_device(device, copied_ >= kWorth);
    if (!pool_ && copied_ >= kWorth) copied_ = 0;  // cannot be had: asked for again after as much
    return pool_ != nullptr;
  }

  // (after wanted() said so) n bytes of host memory to the device, chunk by chunk through fill(pinned, offset, bytes); returns when done. The
  // caller has synchronised the last use of dst.
  template <typename Fill>
  cudaError_t fill_device(void* dst, std::size_t n, int device, Fill&& fill) {
    return run(n, device, [&](Worker& w, std::atomic<std::size_t>& next, std::size_t chunks) {
      int b = 0;
      for (std::size_t i = next++; i < chunks; i = next++, b ^= 1) {
        const std::size_t first = i * kChunk, m = std::min(kChunk, n - first);
        if (const cudaError_t e = cudaEventSynchronize(w.done[b])) return e;
        fill(w.buffer[b], first, m);
        if (const cudaError_t e = cudaMemcpyAsync(static_cast<char*>(dst) + first, w.buffer[b], m, cudaMemcpyHostToDevice, w.stream)) return e;
        if (const cudaError_t e = cudaEventRecord(w.done[b], w.stream)) return e;
      }
      return cudaStreamSynchronize(w.stream);
    });
  }
  // n bytes of device memory, chunk by chunk through drain(pinned, offset, bytes); returns when done. The caller has
  // synchronised the last write of src.
  template <typename Drain>
  cudaError_t drain_device(const void* src, std::size_t n, int device, Drain&& drain) {
    return run(n, device, [&](Worker& w, std::atomic<std::size_t>& next, std::size_t chunks) {
      std::size_t held = chunks;
      int b = 0;
      auto finish = [&](int buffer) {
        const std::size_t first = held * kChunk;
        if (const cudaError_t e = cudaEventSynchronize(w.done[buffer])) return e;
        drain(w.buffer[buffer], first, std::min(kChunk, n - first));
        return cudaSuccess;
      };
      for (std::size_t i = next++; i < chunks; i = next++, b ^= 1) {
        const std::size_t first = i * kChunk, m = std::min(kChunk, n - first);
        if (const cudaError_t e = cudaMemcpyAsync(w.buffer[b], static_cast<const char*>(src) + first, m, cudaMemcpyDeviceToHost, w.stream)) return e;
        if (const cudaError_t e = cudaEventRecord(w.done[b], w.stream)) return e;
        if (held < chunks)
          if (const cudaError_t e = finish(b ^ 1)) return e;
        held = i;
      }
      return held < chunks ? finish(b ^ 1) : cudaSuccess;
    });
  }
  cudaError_t to_device(const void* src, void* dst, std::size_t n, int device) {
    return fill_device(dst, n, device, [&](void* p, std::size_t at, std::size_t m) { std::memcpy(p, static_cast<const char*>(src) + at, m); });
  }
  cudaError_t to_host(const void* src, void* dst, std::size_t n, int device) {
    return drain_device(src, n, device, [&](const void* p, std::size_t at, std::size_t m) { std::memcpy(static_cast<char*>(dst) + at, p, m); });
  }

 private:
  template <typename F>
  cudaError_t run(std::size_t n, int device, F&& body) {
    std::lock_guard<std::mutex> lock(pool_->busy);
    std::vector<Worker>& workers_ = pool_->workers;
    const std::size_t chunks = (n + kChunk - 1) / kChunk;
    std::atomic<std::size_t> next{0};
    std::vector<cudaError_t> status(workers_.size(), cudaSuccess);
    auto work = [&](std::size_t k) {
      status[k] = cudaSetDevice(device);
      if (status[k] == cudaSuccess) status[k] = body(workers_[k], next, chunks);
      if (status[k] != cudaSuccess) next = chunks;  // the others stop after their chunk
    };
    std::vector<std::thread> threads;
    threads.reserve(workers_.size());
    try {
      for (std::size_t k = 1; k < std::min(workers_.size(), chunks); ++k) threads.emplace_back(work, k);
    } catch (const std::exception&) {  // fewer threads: the others take their chunks
    }
    work(0);
    for (std::thread& t : threads) t.join();
    cudaError_t e = cudaSuccess;
    for (std::size_t k = 0; k < workers_.size(); ++k) {
      if (e == cudaSuccess) e = status[k];
      if (status[k] != cudaSuccess) cudaStreamSynchronize(workers_[k].stream);  // no copy of this call is left in flight
    }
    return e;
  }

  std::shared_ptr<CopyPool> pool_;
  std::size_t copied_ = 0;  // host bytes copied without it that would have taken this path
};

// Wave packets: n complex128 on the host, complex128 or complex64 on the device.
template <typename T>
class HostCopier {
 public:
  using V = std::conditional_t<sizeof(T) == 4, float2, double2>;
  bool wanted(const void* p, long long n, int device) { return raw_.wanted(p, sizeof(double2) * static_cast<std::size_t>(n), device); }
  cudaError_t to_device(const double* src, V* dst, long long n, int device) {
    if constexpr (sizeof(T) == 8) return raw_.to_device(src, dst, sizeof(V) * n, device);
    else
      return raw_.fill_device(dst, sizeof(V) * n, device, [&](void* p, std::size_t at, std::size_t m) {
        float* const q = static_cast<float*>(p);
        const double* const s = src + at / sizeof(float);
        for (std::size_t k = 0; k < m / sizeof(float); ++k) q[k] = static_cast<float>(s[k]);
      });
  }
  cudaError_t to_host(const V* src, double* dst, long long n, int device) {
    if constexpr (sizeof(T) == 8) return raw_.to_host(src, dst, sizeof(V) * n, device);
    else
      return raw_.drain_device(src, sizeof(V) * n, device, [&](const void* p, std::size_t at, std::size_t m) {
        const float* const q = static_cast<const float*>(p);
        double* const d = dst + at / sizeof(float);
        for (std::size_t k = 0; k < m / sizeof(float); ++k) d[k] = q[k];
      });
  }

 private:
  RawCopier raw_;
};

}  // namespace spo_host
