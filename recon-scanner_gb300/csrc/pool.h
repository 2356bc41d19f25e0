// pool.h -- working memory of calls, from one CUDA memory pool per device.
//
// A call's scratch arrays lived and died with it: 110 us for each cudaMalloc and
// cudaFree pair (450 us at half a gigabyte), which was most of a short call.
// Allocations from the pool are ordered on the stream that uses them (the driver
// orders their reuse on another stream) and cost a few microseconds.  What the
// process keeps between calls is bounded by kPoolKeepBytes; the driver gives the
// rest back whenever a stream synchronises.  What is kept goes back too when the
// device's last context or TSDF volume goes (PoolUser), and when an allocation of
// this library finds the device full (alloc_or_give_back).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <mutex>

namespace rmvs {

constexpr unsigned long long kPoolKeepBytes = 1ull << 30;

constexpr int kMaxDevices = 64;

// The device's pool, made on first use and kept for the life of the process
// (allocations may outlive the thread that made them).
inline cudaError_t scratch_pool(int device, cudaMemPool_t* out) {
  static std::mutex mu;
  static cudaMemPool_t pools[kMaxDevices] = {};
  if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lk(mu);
  if (!pools[device]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaMemPool_t p = nullptr;
    cudaError_t e = cudaMemPoolCreate(&p, &props);
    if (e != cudaSuccess) return e;
    unsigned long long keep = kPoolKeepBytes;
    e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) {
      cudaMemPoolDestroy(p);
      return e;
    }
    pools[device] = p;
  }
  *out = pools[device];
  return cudaSuccess;
}

// Returns the pool's unused memory to the device; frees still in a stream's queue
// stay, unless `wait` lets them finish first.
inline void pool_give_back(int device, bool wait) {
  cudaMemPool_t pool;
  if (wait) cudaDeviceSynchronize();
  if (scratch_pool(device, &pool) == cudaSuccess) cudaMemPoolTrimTo(pool, 0);
}

// Runs `alloc` (a cudaError_t()); where the device is full, once more without what
// the pool keeps.
template <class F>
cudaError_t alloc_or_give_back(F alloc) {
  cudaError_t e = alloc();
  int device = 0;
  if (e != cudaErrorMemoryAllocation || cudaGetDevice(&device) != cudaSuccess) return e;
  cudaGetLastError();
  pool_give_back(device, true);
  return alloc();
}

// Counts what holds arrays of a device's pool, its contexts and TSDF volumes; the
// last one to go gives the pool's memory back.
class PoolUser {
  int device_ = -1;
  static std::atomic<int>& users(int device) {
    static std::atomic<int> n[kMaxDevices];
    return n[device];
  }

 public:
  PoolUser() = default;
  PoolUser(const PoolUser&) = delete;
  PoolUser& operator=(const PoolUser&) = delete;
  void join(int device) {
    if (device < 0 || device >= kMaxDevices) return;
    device_ = device;
    ++users(device);
  }
  ~PoolUser() {
    if (device_ >= 0 && --users(device_) == 0) pool_give_back(device_, false);
  }
};

// An array with an allocation of its own, for what is large and lives long: where
// the pool has nothing kept, mapping and unmapping through it takes 2.3 us a
// megabyte (372 MB: 0.85 ms), an allocation of its own 1.2.  Freed at once, after
// the device's work.
template <class T>
struct OwnArray {
  T* p = nullptr;
  size_t n = 0;
  OwnArray() = default;
  OwnArray(const OwnArray&) = delete;
  OwnArray& operator=(const OwnArray&) = delete;
  ~OwnArray() { release(); }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
  // At least `count` elements; a larger array does not keep the old contents.
  cudaError_t reserve(size_t count) {
    if (count <= n && p) return cudaSuccess;
    release();
    const cudaError_t e =
        alloc_or_give_back([&] { return cudaMalloc((void**)&p, std::max<size_t>(count, 1) * sizeof(T)); });
    if (e != cudaSuccess) {
      p = nullptr;
      return e;
    }
    n = count;
    return cudaSuccess;
  }
};

// An array of the pool, used on one stream only; freed in that stream's order.
template <class T>
struct PoolArray {
  T* p = nullptr;
  size_t n = 0;
  int device = 0;
  cudaStream_t stream = nullptr;
  PoolArray() = default;
  PoolArray(int device_, cudaStream_t stream_) : device(device_), stream(stream_) {}
  PoolArray(const PoolArray&) = delete;
  PoolArray& operator=(const PoolArray&) = delete;
  ~PoolArray() { release(); }
  void release() {
    if (p) cudaFreeAsync(p, stream);
    p = nullptr;
    n = 0;
  }
  // At least `count` elements; a larger array does not keep the old contents.
  cudaError_t reserve(size_t count) {
    if (count <= n && p) return cudaSuccess;
    release();
    cudaMemPool_t pool;
    cudaError_t e = scratch_pool(device, &pool);
    if (e == cudaSuccess)
      e = alloc_or_give_back(
          [&] { return cudaMallocFromPoolAsync((void**)&p, std::max<size_t>(count, 1) * sizeof(T), pool, stream); });
    if (e != cudaSuccess) {
      p = nullptr;
      return e;
    }
    n = count;
    return cudaSuccess;
  }
};

}  // namespace rmvs
