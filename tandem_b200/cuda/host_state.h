// What launches on one GPU share on the host.  Several threads launch at once (autograd's workers, an evaluation beside a
// training step), so whatever is made by the first call or handed out from call to call sits behind a lock or is atomic.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <mutex>

namespace tb {

// SMs of the GPU; 0 where there is none.
inline int sm_count() {
  static std::atomic<int> known{0};
  int n = known.load(std::memory_order_relaxed);
  if (n == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 0) n = 0;
    cudaGetLastError();
    known.store(n, std::memory_order_relaxed);
  }
  return n;
}

// The dynamic shared memory that a kernel may ask for, raised before its first launch on each device: the limit belongs to the
// device.  Only a success is remembered.
class SharedMemoryLimit {
 public:
  template <typename... Args>
  cudaError_t raise(void (*kernel)(Args...), int bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
    if (raised_.load(std::memory_order_relaxed) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) raised_.fetch_or(bit, std::memory_order_relaxed);
    else cudaGetLastError();  // it is returned: the next launch does not find it again
    return e;
  }

 private:
  std::atomic<unsigned long long> raised_{0};
};

// A word of host memory that kernels raise when a wait runs out.
class ErrorWord {
 public:
  bool raised() const {
    const int* word = host_.load(std::memory_order_acquire);
    return word != nullptr && *reinterpret_cast<const volatile int*>(word) != 0;
  }
  // Its device address; null if it cannot be made.
  int* device() {
    if (host_.load(std::memory_order_acquire) != nullptr) return dev_;
    std::lock_guard<std::mutex> hold(lock_);
    if (host_.load(std::memory_order_relaxed) != nullptr) return dev_;
    int *host = nullptr, *dev = nullptr;
    if (cudaHostAlloc((void**)&host, 64, cudaHostAllocMapped) != cudaSuccess) return nullptr;
    *host = 0;
    if (cudaHostGetDevicePointer((void**)&dev, host, 0) != cudaSuccess) {
      cudaFreeHost(host);
      return nullptr;
    }
    dev_ = dev;
    host_.store(host, std::memory_order_release);  // last: whoever sees it sees dev_
    return dev;
  }

 private:
  std::mutex lock_;
  std::atomic<int*> host_{nullptr};
  int* dev_ = nullptr;
};

// Words of a __device__ array of 2 * `size` zeros, lent round-robin to launches that leave them zero again: launches in flight at
// the same time share none (`size` words' worth of them would have to overlap).  A launch that is recorded into a graph keeps its
// words for every replay, so those come from the second half: whatever is issued beside a replay has others.  Two graphs that are
// replayed at the same time may share words, if between their recordings a whole half was lent.
class WordPool {
 public:
  explicit WordPool(long long size) : size_(size) {}
  // `words` <= size of them for a launch on `stream` of the current device; `find(void**)` looks the array up there.
  template <typename Find>
  cudaError_t take(long long words, cudaStream_t stream, unsigned** out, Find find) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) {  // the launch itself will meet the reason
      cudaGetLastError();
      status = cudaStreamCaptureStatusNone;
    }
    const int half = status != cudaStreamCaptureStatusNone;
    std::lock_guard<std::mutex> hold(lock_);
    if (device_ != dev) {
      void* at = nullptr;
      if ((e = find(&at)) != cudaSuccess) return e;
      pool_ = static_cast<unsigned*>(at);
      device_ = dev;
    }
    if (next_[half] + words > size_) next_[half] = 0;
    *out = pool_ + half * size_ + next_[half];
    next_[half] += words;
    return cudaSuccess;
  }

 private:
  std::mutex lock_;
  const long long size_;
  unsigned* pool_ = nullptr;
  int device_ = -1;
  long long next_[2] = {0, 0};
};

}  // namespace tb
