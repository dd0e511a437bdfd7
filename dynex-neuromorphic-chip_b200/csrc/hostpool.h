// Helper threads for host passes over large arrays, and copies between pageable host memory
// and the device through them.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <functional>

namespace dmm {

// Runs f(part) for part = 0 .. parts-1 on the calling thread and up to kPoolHelpers helper
// threads of the process, and returns when all are done.  One call at a time uses the helpers;
// a call that finds them busy (or a forked child, which has none) runs its parts itself.
constexpr int kPoolHelpers = 7;
void pool_run(int parts, const std::function<void(int)>& f);
// Parts for a pass over `bytes` of memory: one per 128 KB, at most the helpers and the caller.
int pool_parts(int64_t bytes);

// Copies between a caller's pageable array and device memory, chunk by chunk through
// page-locked buffers that the pool fills or empties.  The driver's own pageable copies move
// 6-11 GB/s on one thread, and a fresh destination array costs it a page fault every 4 KB; the
// pool's threads share both, and FP32 states cross as floats.  n = 10^6, m = 8 10^6 (136 MB of
// doubles): state upload 12.2 -> 4.0 ms, state read 29.6 -> 7.9 ms; n = 20,000, m = 86,000 in
// FP64: a right-hand side and an Euler step with their copies 1,020 -> 430 us.
class HostXfer {
 public:
  ~HostXfer();
  // count doubles at src to dst as T (float: rounded to nearest, as on the device), queued on
  // s; src is read when the call returns.
  template <class T>
  cudaError_t upload(T* dst, const double* src, int64_t count, cudaStream_t s);
  // count T at src to doubles at dst; waits for s.
  template <class T>
  cudaError_t download(double* dst, const T* src, int64_t count, cudaStream_t s);

 private:
  static constexpr int kBufs = 4;
  static constexpr int64_t kBytes = int64_t(1) << 20;
  struct Buf {
    unsigned char* p = nullptr;
    cudaEvent_t done = nullptr;
    bool busy = false;
  };
  cudaError_t ready(Buf& b);
  Buf buf_[kBufs];
  int next_ = 0;
};

// A HostXfer of the current device for the scope of a call: taken from the idle ones of the
// process (one per device and concurrent caller, 4 MB each) and put back; its last copies may
// still be on their way then, and the next user waits for the buffers it needs.
class XferLease {
 public:
  XferLease();
  ~XferLease();
  HostXfer* operator->() const { return x_; }

 private:
  HostXfer* x_;
  int dev_;
};
// Frees the idle ones.
void release_xfers();

}  // namespace dmm
