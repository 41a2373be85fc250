// Host waits that sleep.  cudaStreamSynchronize spins a core for the whole wait (the default
// scheduling of a context that has fewer threads than cores); a caller with several extractions
// in flight, or a request server, has many threads waiting at once, and their spinning takes the
// host's cores from the threads that have work.  A blocking-sync event (one per thread and device)
// puts the waiting thread to sleep instead.  A sleeping thread takes some 20 us to come back, which a
// small extraction would pay three times in a call of 200 us; so a wait polls for its first 60 us and
// sleeps after that.
#pragma once
#include <chrono>
#include <vector>
#include <cuda_runtime.h>

namespace tmc {

// Marks the work queued on `st` so far, for host_wait_mark on the same thread (before its next mark).
// The event belongs to the current device; null when it cannot be recorded on `st` (a stream of another
// device, or an event left from before a device reset, which is replaced once).
inline cudaEvent_t host_mark(cudaStream_t st) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  thread_local std::vector<cudaEvent_t> events;  // by device
  if ((int)events.size() <= dev) events.resize(dev + 1, nullptr);
  for (int attempt = 0; attempt < 2; attempt++) {
    if (!events[dev] &&
        cudaEventCreateWithFlags(&events[dev], cudaEventBlockingSync | cudaEventDisableTiming) != cudaSuccess) {
      (void)cudaGetLastError();
      events[dev] = nullptr;
      break;
    }
    if (cudaEventRecord(events[dev], st) == cudaSuccess) return events[dev];
    (void)cudaGetLastError();
    events[dev] = nullptr;
  }
  return nullptr;
}

// Waits for the marked work; without a mark, for all of the stream's.
inline cudaError_t host_wait_mark(cudaEvent_t mark, cudaStream_t st) {
  if (!mark) return cudaStreamSynchronize(st);
  // a query that is not ready yet counts as the thread's last error: poll only when there is none to
  // lose, and take each one back
  if (cudaPeekAtLastError() == cudaSuccess) {
    const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(60);
    do {
      const cudaError_t e = cudaEventQuery(mark);
      if (e != cudaErrorNotReady) return e;
      (void)cudaGetLastError();
    } while (std::chrono::steady_clock::now() < until);
  }
  return cudaEventSynchronize(mark);
}

// Waits for the work queued on `st` so far.
inline cudaError_t host_wait(cudaStream_t st) { return host_wait_mark(host_mark(st), st); }

}  // namespace tmc
