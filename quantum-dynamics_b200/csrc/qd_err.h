// qd_err.h -- error reporting and call scratch shared by the library's
// translation units.
#pragma once
#include <cstdarg>
#include <cstdio>
#include <cuda_runtime.h>
#include "qd.h"

int qd_set_error(int code, const char *msg);     // sets qd_last_error(), returns code
void qd_count_launches(int n);                    // qd_kernel_launch_count bookkeeping

inline int qd_errf(int code, const char *fmt, ...)
{
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  return qd_set_error(code, buf);
}

#define QD_CU(x)                                                                        \
  do {                                                                                  \
    cudaError_t e_ = (x);                                                               \
    if (e_ != cudaSuccess)                                                              \
      return qd_errf(QD_ERR_CUDA, "%s failed: %s (%s:%d)", #x, cudaGetErrorString(e_),   \
                     __FILE__, __LINE__);                                               \
  } while (0)

// Device memory of one call (the set-up entry points, which work on the legacy
// default stream): allocated on construction, returned to the pool on
// destruction, in stream order.  The pool keeps at most QD_SCRATCH_KEEP bytes
// between calls and belongs to the current device, so a call does not pay
// cudaMalloc and cudaFree (0.2-0.5 ms together, and a device-wide wait).
constexpr size_t QD_SCRATCH_KEEP = size_t(256) << 20;
cudaError_t qd_scratch_alloc(void **p, size_t bytes);
// device -> host on the legacy default stream, through the page-locked staging
// buffers and the host threads from 2 MB on (a fresh result array's page faults
// are then shared by the threads too); returns when dst holds the data
cudaError_t qd_fetch(void *dst, const void *src, size_t bytes);
struct qd_scratch {
  void *p = nullptr;
  size_t bytes;
  explicit qd_scratch(size_t n) : bytes(n)
  {
    if (qd_scratch_alloc(&p, n) != cudaSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
  }
  ~qd_scratch()
  {
    if (p) cudaFreeAsync(p, 0);
  }
  qd_scratch(const qd_scratch &) = delete;
  qd_scratch &operator=(const qd_scratch &) = delete;
  template <typename T> T *at() const { return static_cast<T *>(p); }
};
