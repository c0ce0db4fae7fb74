/* The few calls of the CUDA runtime that host_copy.h makes, on the host: copies
   are made at once, an event completes when the work queued before it would
   (fake::busy_until), and page-locked memory is counted and can be refused. */
#ifndef FAKE_CUDA_RUNTIME_H
#define FAKE_CUDA_RUNTIME_H

#include <chrono>
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <set>
#include <thread>

typedef int cudaError_t;
typedef int cudaStream_t;
enum { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorInvalidValue = 1 };
enum { cudaMemcpyDeviceToHost = 2, cudaHostAllocPortable = 1, cudaEventDisableTiming = 2 };
enum { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1 };
struct cudaPointerAttributes {
  int type;
};

namespace fake {
typedef std::chrono::steady_clock clock;
inline clock::time_point busy_until;
inline std::set<void*> locked;
inline int allocs = 0, frees = 0, last_error = cudaSuccess;
inline bool refuse = false;
inline int set(int e) {
  if (e) last_error = e;
  return e;
}
}  // namespace fake

struct FakeEvent {
  fake::clock::time_point at;
};
typedef FakeEvent* cudaEvent_t;

inline cudaError_t cudaGetLastError() {
  const int e = fake::last_error;
  fake::last_error = cudaSuccess;
  return e;
}
inline cudaError_t cudaHostAlloc(void** p, size_t n, int) {
  if (fake::refuse) return fake::set(cudaErrorMemoryAllocation);
  fake::allocs++;
  fake::locked.insert(*p = std::malloc(n));
  return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void* p) {
  if (!fake::locked.erase(p)) return fake::set(cudaErrorInvalidValue);
  fake::frees++;
  std::free(p);
  return cudaSuccess;
}
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* at, const void* p) {
  at->type = fake::locked.count(const_cast<void*>(p)) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, int, cudaStream_t) {
  std::memcpy(dst, src, n);
  return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t) {
  std::this_thread::sleep_until(fake::busy_until);
  return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, int) {
  *e = new FakeEvent;
  return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete e;
  return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
  e->at = fake::busy_until;
  return cudaSuccess;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  std::this_thread::sleep_until(e->at);
  return cudaSuccess;
}

#endif
