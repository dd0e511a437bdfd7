// Helper threads and chunked host copies (hostpool.h).
#include "hostpool.h"

#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

#include "devmem.h"

namespace dmm {
namespace {

class Pool {
 public:
  ~Pool() {
    {
      std::lock_guard<std::mutex> g(mu_);
      stop_ = true;
    }
    cv_.notify_all();
    for (auto& t : threads_) t.join();
  }
  bool own_process() const { return getpid() == pid_; }

  void run(int parts, const std::function<void(int)>& f) {
    std::unique_lock<std::mutex> user(user_mu_, std::try_to_lock);
    if (parts <= 1 || !user.owns_lock() || !start()) {
      for (int i = 0; i < parts; i++) f(i);
      return;
    }
    {
      std::lock_guard<std::mutex> g(mu_);
      f_ = &f;
      parts_ = parts;
      taken_.store(0);
      left_.store(parts);
      in_.store(0);
      epoch_.fetch_add(1);
    }
    cv_.notify_all();
    work(&f, parts);
    // the parts are short: wait for the helpers that took one
    while (left_.load(std::memory_order_acquire) > 0) std::this_thread::yield();
    std::lock_guard<std::mutex> g(mu_);
    f_ = nullptr;
    while (in_.load(std::memory_order_acquire) > 0) std::this_thread::yield();
  }

 private:
  bool start() {
    if (!own_process()) return false;
    if (!threads_.empty()) return true;
    const int hw = (int)std::thread::hardware_concurrency();
    const int want = std::min(kPoolHelpers, hw - 1);
    try {
      for (int i = 0; i < want; i++) threads_.emplace_back([this] { loop(); });
    } catch (...) {
    }
    return !threads_.empty();
  }

  void work(const std::function<void(int)>* f, int parts) {
    for (;;) {
      const int i = taken_.fetch_add(1);
      if (i >= parts) break;
      (*f)(i);
      left_.fetch_sub(1, std::memory_order_release);
    }
  }

  void loop() {
    uint64_t seen = 0;
    for (;;) {
      // calls often follow one another: look for the next one briefly before sleeping
      const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(60);
      while (epoch_.load(std::memory_order_acquire) == seen &&
             std::chrono::steady_clock::now() < until)
        std::this_thread::yield();
      const std::function<void(int)>* f = nullptr;
      int parts = 0;
      {
        std::unique_lock<std::mutex> g(mu_);
        cv_.wait(g, [&] { return stop_ || epoch_.load() != seen; });
        if (stop_) return;
        seen = epoch_.load();
        f = f_;
        parts = parts_;
        if (f) in_.fetch_add(1);
      }
      if (!f) continue;  // the call ended before this thread woke
      work(f, parts);
      in_.fetch_sub(1, std::memory_order_release);
    }
  }

  const pid_t pid_ = getpid();
  std::mutex user_mu_, mu_;
  std::condition_variable cv_;
  std::vector<std::thread> threads_;
  const std::function<void(int)>* f_ = nullptr;
  int parts_ = 0;
  bool stop_ = false;
  std::atomic<uint64_t> epoch_{0};
  std::atomic<int> taken_{0}, left_{0}, in_{0};
};

// Ended with the process.  A forked child has none of the threads but a copy of their state, where
// they still wait: destroying the condition variable there would wait for them for ever, so the
// child leaves the pool as it is.
struct PoolOwner {
  Pool* const p = new Pool;
  ~PoolOwner() {
    if (p->own_process()) delete p;
  }
};

Pool& pool() {
  static PoolOwner o;
  return *o.p;
}

constexpr int64_t kTouchBytes = int64_t(4) << 20;

// memcpy, or the conversion between double and float, of [lo, hi).
inline void convert(double* d, const double* s, int64_t lo, int64_t hi) {
  std::memcpy(d + lo, s + lo, (size_t)(hi - lo) * sizeof(double));
}
inline void convert(float* d, const double* s, int64_t lo, int64_t hi) {
  for (int64_t i = lo; i < hi; i++) d[i] = (float)s[i];
}
inline void convert(double* d, const float* s, int64_t lo, int64_t hi) {
  for (int64_t i = lo; i < hi; i++) d[i] = (double)s[i];
}

template <class D, class S>
void spread(D* d, const S* s, int64_t count) {
  const int parts = pool_parts(count * (int64_t)(sizeof(D) + sizeof(S)) / 2);
  const int64_t per = ((count + parts - 1) / parts + 511) & ~int64_t(511);  // whole pages
  pool_run(parts, [&](int i) {
    const int64_t lo = std::min(count, i * per), hi = std::min(count, lo + per);
    if (hi > lo) convert(d, s, lo, hi);
  });
}

}  // namespace

void pool_run(int parts, const std::function<void(int)>& f) { pool().run(parts, f); }

int pool_parts(int64_t bytes) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(kPoolHelpers + 1, bytes >> 17));
}

namespace {
struct Idle {
  std::mutex mu;
  std::map<int, std::vector<HostXfer*>> by_dev;
};
Idle& idle() {
  static Idle* i = new Idle;  // (left to the process's end: buffers must outlive every pack)
  return *i;
}
}  // namespace

XferLease::XferLease() : x_(nullptr), dev_(-1) {
  if (cudaGetDevice(&dev_) != cudaSuccess) {
    cudaGetLastError();
    dev_ = -1;
  }
  std::lock_guard<std::mutex> g(idle().mu);
  auto& v = idle().by_dev[dev_];
  if (v.empty()) {
    x_ = new HostXfer;
  } else {
    x_ = v.back();
    v.pop_back();
  }
}

XferLease::~XferLease() {
  std::lock_guard<std::mutex> g(idle().mu);
  idle().by_dev[dev_].push_back(x_);
}

void release_xfers() {
  std::map<int, std::vector<HostXfer*>> all;
  {
    std::lock_guard<std::mutex> g(idle().mu);
    all.swap(idle().by_dev);
  }
  for (auto& kv : all)
    for (HostXfer* x : kv.second) delete x;
}

HostXfer::~HostXfer() {
  for (Buf& b : buf_) {
    if (b.busy) cudaEventSynchronize(b.done);
    if (b.p) pinned_free(b.p);
    if (b.done) cudaEventDestroy(b.done);
  }
}

cudaError_t HostXfer::ready(Buf& b) {
  if (!b.p) {
    void* p = nullptr;
    cudaError_t e = pinned_alloc(&p, kBytes);
    if (e != cudaSuccess) return e;
    b.p = static_cast<unsigned char*>(p);
    e = cudaEventCreateWithFlags(&b.done, cudaEventDisableTiming);
    if (e != cudaSuccess) return e;
  }
  if (b.busy) {
    const cudaError_t e = cudaEventSynchronize(b.done);
    if (e != cudaSuccess) return e;
    b.busy = false;
  }
  return cudaSuccess;
}

template <class T>
cudaError_t HostXfer::upload(T* dst, const double* src, int64_t count, cudaStream_t s) {
  const int64_t per = kBytes / (int64_t)sizeof(T);
  for (int64_t at = 0; at < count; at += per) {
    const int64_t k = std::min(per, count - at);
    Buf& b = buf_[next_];
    next_ = (next_ + 1) % kBufs;
    cudaError_t e = ready(b);
    if (e != cudaSuccess) return e;
    spread(reinterpret_cast<T*>(b.p), src + at, k);
    e = cudaMemcpyAsync(dst + at, b.p, (size_t)k * sizeof(T), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaEventRecord(b.done, s);
    if (e != cudaSuccess) return e;
    b.busy = true;
  }
  return cudaSuccess;
}

template <class T>
cudaError_t HostXfer::download(double* dst, const T* src, int64_t count, cudaStream_t s) {
  const int64_t per = kBytes / (int64_t)sizeof(T);
  const int64_t chunks = (count + per - 1) / per;
  const int first = next_;
  auto at_buf = [&](int64_t c) -> Buf& { return buf_[(first + c) % kBufs]; };
  auto issue = [&](int64_t c) -> cudaError_t {
    Buf& b = at_buf(c);
    cudaError_t e = ready(b);
    if (e != cudaSuccess) return e;
    const int64_t k = std::min(per, count - c * per);
    e = cudaMemcpyAsync(b.p, src + c * per, (size_t)k * sizeof(T), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaEventRecord(b.done, s);
    if (e == cudaSuccess) b.busy = true;
    return e;
  };
  for (int64_t c = 0; c < std::min<int64_t>(chunks, kBufs); c++) {
    const cudaError_t e = issue(c);
    if (e != cudaSuccess) return e;
  }
  // A fresh destination costs a page fault per 4 KB, or 2 MB with huge pages: each thread takes
  // those of its own share (in the chunks below all threads would meet on the same huge page)
  if (count * 8 >= kTouchBytes) {
    const int parts = pool_parts(count * 8);
    volatile char* base = reinterpret_cast<volatile char*>(dst);
    pool_run(parts, [&](int i) {
      const int64_t lo = count * 8 * i / parts, hi = count * 8 * (i + 1) / parts;
      for (int64_t o = lo; o < hi; o += 4096) base[o] = 0;
    });
  }
  for (int64_t c = 0; c < chunks; c++) {
    Buf& b = at_buf(c);
    cudaError_t e = ready(b);  // waits for the chunk
    if (e != cudaSuccess) return e;
    spread(dst + c * per, reinterpret_cast<const T*>(b.p), std::min(per, count - c * per));
    if (c + kBufs < chunks) {
      e = issue(c + kBufs);
      if (e != cudaSuccess) return e;
    }
  }
  next_ = (int)((first + chunks) % kBufs);
  return cudaSuccess;
}

template cudaError_t HostXfer::upload<float>(float*, const double*, int64_t, cudaStream_t);
template cudaError_t HostXfer::upload<double>(double*, const double*, int64_t, cudaStream_t);
template cudaError_t HostXfer::download<float>(double*, const float*, int64_t, cudaStream_t);
template cudaError_t HostXfer::download<double>(double*, const double*, int64_t, cudaStream_t);

}  // namespace dmm
