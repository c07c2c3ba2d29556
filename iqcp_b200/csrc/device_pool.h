// Device memory and streams of the contexts, kept between contexts.
//
// A geometry scan makes and destroys a context per step.  Thirty cudaMalloc and
// cudaFree calls, four streams and a cudaGetDeviceProperties took most of the
// 15 ms an H2O context cost (3 ms with them gone); here a context's arrays are carved out of a few
// blocks, blocks come from a memory pool of the library's own, and streams
// are handed on.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstring>
#include <vector>

namespace iqcp {

// What the library keeps for the process (pool, idle streams, launch limits) ends
// with the device's CUDA context: a caller may reset the device between two
// contexts.  device_refresh, called where a context is made or destroyed with the
// device current, asks for the CUDA context's id, which no later one shares; on a
// new id it forgets what belonged to the old one and counts the epoch on.
cudaError_t device_refresh(int device, unsigned long long* id);
unsigned device_epoch(int device);

// Memory from the library's pool on `device`, ordered on `stream`.  The pool is
// the driver's stream-ordered allocator: safe from several threads and streams,
// and it gives freed memory above kPoolKeep bytes back to the device whenever a
// stream is synchronised.
// Blocks above kPoolMax come from cudaMalloc: the pool would map and unmap them at
// every context, and a context that large is not made to be thrown away.
constexpr unsigned long long kPoolKeep = 64ull << 20, kPoolMax = 16ull << 20;
cudaError_t pool_alloc(int device, void** p, size_t bytes, cudaStream_t stream);
void pool_free(void* p, cudaStream_t stream);

// A small block from cudaMalloc, whose cudaFree waits for all work on the device
// (drain).  A context's calls may have left work on any stream it was given, and
// graphs that captured them may be running: its pooled memory and streams are
// handed on only behind such a wait.  cudaDeviceSynchronize would end every
// capture in progress on the device with an error, that of another thread's
// batched SCF among them.
cudaError_t drain_block(int device, void** p);
cudaError_t drain(void* block);

// Allocation calls of this thread are allowed beside captures while one of these lives
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// Eight non-blocking streams (a small molecule's class kernels are a block or two
// each, and their launches the longer the more of them run at once).  Returned sets are handed on to later contexts of
// the same device, at most kKeepStreams idle sets per device.  A set is returned
// only when its streams are idle.
constexpr int kSetStreams = 8, kKeepStreams = 8;
struct StreamSet {
  cudaStream_t s[kSetStreams] = {};
};
cudaError_t streams_take(int device, StreamSet* set);
void streams_give(int device, const StreamSet& set);

// Arrays of one allocation: want() each, alloc(), and the pointers are set.
// Arrays given with their contents are placed first and uploaded in one copy.
class DeviceBlock {
 public:
  template <typename T>
  void want(T** p, size_t n) {
    add((void**)p, nullptr, sizeof(T) * n);
  }
  template <typename T>
  void upload(T** p, const T* src, size_t n) {
    add((void**)p, src, sizeof(T) * n);
  }
  // Allocates on `stream` and enqueues the upload; the sources are read before it returns.
  cudaError_t alloc(int device, cudaStream_t stream);
  void free(cudaStream_t stream);

 private:
  struct Item {
    void** p;
    const void* src;
    size_t bytes;
  };
  void add(void** p, const void* src, size_t bytes) { items_.push_back({p, src, bytes}); }
  std::vector<Item> items_;
  void* base_ = nullptr;
  bool pooled_ = false;
};

}  // namespace iqcp
