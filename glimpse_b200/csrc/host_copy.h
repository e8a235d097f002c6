// Copies between a caller's ordinary (pageable) host memory and the device, for
// the entry points that move tens of megabytes a call.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <thread>
#include <vector>

namespace gp {

// Pinned staging buffers of one context: made at the first large copy, kept
// (kThreads * kBuffers * kBytes in all) and freed with the context. One host thread
// per context, so no lock.
//
// A pageable copy is staged by the driver on one thread: 12 GB/s in, measured. With
// four threads that fill buffers of their own, the link is the limit.
class HostStage {
 public:
  static constexpr int kThreads = 4, kBuffers = 2;
  static constexpr size_t kBytes = size_t(512) << 10;
  static constexpr size_t kLarge = size_t(8) << 20;  // below, the plain copy is as fast

  // Host to device on a stream. As cudaMemcpyAsync from pageable memory, src may
  // be changed when this returns; copies queued later on the stream come after.
  cudaError_t copy_in(int device, void* dst, const void* src, size_t bytes, cudaStream_t stream);
  void release();

 private:
  bool ready = false;
  char* pinned = nullptr;
  cudaEvent_t done[kThreads][kBuffers] = {};
  cudaError_t make();
};

// Backs the pages of an output buffer while the device works: the first write to
// fresh memory faults page by page, three quarters of the time of a copy into it
// (16.4 against 3.6 ms for 77 MB). Contents are not changed; memory that is backed
// already, or a system without the request, costs nothing.
class Prefault {
 public:
  Prefault() = default;
  Prefault(const Prefault&) = delete;
  Prefault& operator=(const Prefault&) = delete;
  ~Prefault() { wait(); }
  void start(void* p, size_t bytes);
  void wait();

 private:
  std::vector<std::thread> threads;
};

}  // namespace gp
