// Staged copies of pageable host memory (host_copy.h).
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstdint>
#include <cstring>

#include "host_copy.h"

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23
#endif

namespace gp {

cudaError_t HostStage::make() {
  if (ready) return cudaSuccess;
  cudaError_t e = cudaMallocHost(reinterpret_cast<void**>(&pinned), kThreads * kBuffers * kBytes);
  if (e != cudaSuccess) {
    pinned = nullptr;
    return e;
  }
  for (auto& row : done)
    for (auto& ev : row)
      if ((e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming)) != cudaSuccess) return e;
  ready = true;
  return cudaSuccess;
}

void HostStage::release() {
  for (auto& row : done)
    for (auto& ev : row) {
      if (ev) {
        cudaEventSynchronize(ev);
        cudaEventDestroy(ev);
      }
      ev = nullptr;
    }
  if (pinned) cudaFreeHost(pinned);
  pinned = nullptr;
  ready = false;
}

// Whether memory is ordinary (the driver copies pinned or managed memory straight from where it is).
static bool pageable(const void* p) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, p) == cudaSuccess) return at.type == cudaMemoryTypeUnregistered;
  cudaGetLastError();
  return false;
}

cudaError_t HostStage::copy_in(int device, void* dst, const void* src, size_t bytes, cudaStream_t stream) {
  bool staged = bytes >= kLarge && pageable(src);
  if (staged && make() != cudaSuccess) {
    cudaGetLastError();  // no pinned memory to be had: the plain copy does
    release();
    staged = false;
  }
  if (!staged) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, stream);
  cudaError_t err[kThreads] = {};
  // thread i takes the pieces i, i + kThreads, ...
  auto work = [&](int i) {
    cudaError_t e = cudaSetDevice(device);
    int b = 0;
    for (size_t o = i * kBytes; o < bytes && e == cudaSuccess; o += kThreads * kBytes, b = (b + 1) % kBuffers) {
      char* p = pinned + (size_t)(i * kBuffers + b) * kBytes;
      const size_t n = std::min(kBytes, bytes - o);
      if ((e = cudaEventSynchronize(done[i][b])) != cudaSuccess) break;  // its last copy; at once if there was none
      std::memcpy(p, static_cast<const char*>(src) + o, n);
      e = cudaMemcpyAsync(static_cast<char*>(dst) + o, p, n, cudaMemcpyHostToDevice, stream);
      if (e == cudaSuccess) e = cudaEventRecord(done[i][b], stream);
    }
    err[i] = e;
  };
  std::thread t[kThreads];
  int started = 1;  // the caller's thread works too
  try {
    for (; started < kThreads; ++started) t[started] = std::thread(work, started);
  } catch (...) {
  }
  work(0);
  for (int i = 1; i < started; ++i) t[i].join();
  for (int i = started; i < kThreads; ++i) work(i);  // a thread that could not be made
  for (cudaError_t e : err)
    if (e != cudaSuccess) return e;
  return cudaSuccess;
}

void Prefault::start(void* p, size_t bytes) {
  constexpr size_t kMin = size_t(2) << 20;
  if (bytes < kMin || !pageable(p)) return;  // pinned pages are backed: 1.4 ms of looking at 230 MB of them
  const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
  const uintptr_t a = (uintptr_t)p & ~(page - 1), b = ((uintptr_t)p + bytes + page - 1) & ~(page - 1);
  const int n = bytes >= 8 * kMin ? 4 : 1;
  const uintptr_t step = ((b - a) / n + page - 1) & ~(page - 1);
  try {
    for (uintptr_t lo = a; lo < b; lo += step) {
      const uintptr_t hi = std::min(b, lo + step);
      threads.emplace_back([lo, hi] { madvise(reinterpret_cast<void*>(lo), hi - lo, MADV_POPULATE_WRITE); });
    }
  } catch (...) {
    // the copy itself backs what is left
  }
}

void Prefault::wait() {
  for (auto& t : threads) t.join();
  threads.clear();
}

}  // namespace gp
