// The part of the CUDA runtime that qd_staging.h calls, on the host: devices
// that only have a number, streams and events that belong to one, copies done at
// the call.  For tests of the host code where no GPU or only one is present.
#pragma once
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <functional>

enum cudaError_t {
  cudaSuccess = 0,
  cudaErrorInvalidValue = 1,
  cudaErrorMemoryAllocation = 2,
  cudaErrorInvalidDevice = 101,
  cudaErrorInvalidResourceHandle = 400
};
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
enum { cudaHostAllocPortable = 1, cudaEventDisableTiming = 2 };

struct FakeHandle { int dev; };
typedef FakeHandle *cudaStream_t;      // null: the current device's default stream
typedef FakeHandle *cudaEvent_t;

namespace fake {
constexpr int DEVICES = 4;
inline thread_local int device = 0;
inline std::atomic<long> pinned{0};                   // page-locked bytes
inline std::function<void()> on_stream_sync;          // runs inside cudaStreamSynchronize
inline int of(cudaStream_t s) { return s ? s->dev : device; }
}

inline cudaError_t cudaGetDevice(int *d) { *d = fake::device; return cudaSuccess; }
inline cudaError_t cudaSetDevice(int d)
{
  if (d < 0 || d >= fake::DEVICES) return cudaErrorInvalidDevice;
  fake::device = d;
  return cudaSuccess;
}
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaHostAlloc(void **p, size_t n, unsigned)
{
  *p = std::malloc(n);
  fake::pinned += (long)n;
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned)
{
  *e = new FakeHandle{fake::device};
  return cudaSuccess;
}
// an event is recorded on streams of the device it was created on
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
  return e && e->dev == fake::of(s) ? cudaSuccess : cudaErrorInvalidResourceHandle;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
  return e ? cudaSuccess : cudaErrorInvalidResourceHandle;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t)
{
  if (fake::on_stream_sync) fake::on_stream_sync();
  return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
  std::memcpy(d, s, n);
  return cudaSuccess;
}
inline cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k)
{
  const cudaError_t e = cudaMemcpyAsync(d, s, n, k, nullptr);
  return e == cudaSuccess ? cudaStreamSynchronize(nullptr) : e;
}
