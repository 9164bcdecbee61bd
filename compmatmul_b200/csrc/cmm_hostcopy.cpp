// Copies between device memory and caller-owned host memory for the
// host-pointer entry points (the drop-in's matmul_fft / matmul_fwht pass
// ordinary pageable numpy arrays, compmatmul.cpp:107-147).
//
// Page-locked host memory is copied directly with cudaMemcpyAsync.  For
// pageable memory the driver stages the copy through its own pinned buffer
// on one host thread, well below the link's bandwidth; here it goes through
// a ring of pinned slots that several host threads fill (host to device) or
// drain (device to host) at once, while the DMA of the previous slot runs.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

#include "cmm_internal.h"

namespace cmm {
namespace {

// memcpy in equal parts by the caller and a few helpers, for the copies of 256 KB
// to 12 MB that a call on host arrays makes one after another.  A helper stays
// awake for 300 us after a copy, so those that follow in the call find it running;
// the caller takes what parts are left, so one that sleeps costs a wake-up only.
// (Waking helpers for every part of 512 KB made these copies slower than one
// thread's and scattered: calls of 3738 x 179 x 276, b = 16384 on numpy arrays took
// 2.2 to 2.6 ms, with copies by one thread 1.4, now 0.82; 1793 x 97 x 978 0.9 to 1.9,
// 1.4, 0.71; 512-square 0.52, 0.60, 0.38.)
class NearCopy {
 public:
  static constexpr size_t kMin = (size_t)256 << 10, kMax = (size_t)12 << 20;
  static NearCopy& get() {
    static NearCopy* c = new NearCopy();  // lives until exit (threads detach)
    return *c;
  }

  void copy(void* dst, const void* src, size_t n) {
    std::unique_lock<std::mutex> mine(use_, std::try_to_lock);
    if (!mine || helpers_ == 0) {  // the helpers are another thread's
      std::memcpy(dst, src, n);
      return;
    }
    dst_ = static_cast<char*>(dst);
    src_ = static_cast<const char*>(src);
    n_ = n;
    part_ = (n / (helpers_ + 1) + 4096) & ~(size_t)4095;
    const uint64_t parts = (n + part_ - 1) / part_;
    left_.store((unsigned)parts, std::memory_order_relaxed);
    const uint64_t t = ++generation_ << 16 | parts << 8;
    ticket_.store(t);
    if (asleep_.load()) {  // (a helper counts itself before it looks at the ticket for the last time)
      std::lock_guard<std::mutex> g(mu_);
      cv_.notify_all();
    }
    take(t >> 16);
    while (left_.load(std::memory_order_acquire)) std::this_thread::yield();  // parts that helpers copy
  }

 private:
  NearCopy() {
    helpers_ = std::min(std::thread::hardware_concurrency() / 4, 3u);
    for (unsigned i = 0; i < helpers_; ++i) std::thread([this] { run(); }).detach();
  }

  // parts of a copy until all are taken.  The ticket holds its number, its parts and
  // the next one to take: a part is taken only while its copy waits for it.
  void take(uint64_t generation) {
    uint64_t t = ticket_.load();
    while (t >> 16 == generation && (t & 255) < (t >> 8 & 255)) {
      if (!ticket_.compare_exchange_weak(t, t + 1)) continue;
      const size_t off = (size_t)(t & 255) * part_;
      std::memcpy(dst_ + off, src_ + off, std::min(part_, n_ - off));
      left_.fetch_sub(1, std::memory_order_release);
      t = ticket_.load();
    }
  }

  void run() {
    using Clock = std::chrono::steady_clock;
    uint64_t seen = 0;
    for (auto awake = Clock::now();;) {
      const uint64_t generation = ticket_.load() >> 16;
      if (generation != seen) {
        take(seen = generation);
        awake = Clock::now();
      } else if (Clock::now() - awake > std::chrono::microseconds(300)) {
        std::unique_lock<std::mutex> lk(mu_);
        asleep_.fetch_add(1);
        cv_.wait(lk, [&] { return ticket_.load() >> 16 != seen; });
        asleep_.fetch_sub(1);
      } else {
        std::this_thread::yield();
      }
    }
  }

  std::mutex use_, mu_;
  std::condition_variable cv_;
  std::atomic<uint64_t> ticket_{0};
  std::atomic<unsigned> left_{0}, asleep_{0};
  uint64_t generation_ = 0;
  char* dst_ = nullptr;
  const char* src_ = nullptr;
  size_t n_ = 0, part_ = 1;
  unsigned helpers_ = 0;
};

// memcpy split over a small persistent pool of host threads (larger copies: 16 MB in
// four parts take 1.05 times as long in a call of 8000 x 2000 x 8000)
class CopyPool {
 public:
  static CopyPool& get() {
    static CopyPool* pool = new CopyPool();  // lives until exit (threads detach)
    return *pool;
  }

  void copy(void* dst, const void* src, size_t n) {
    if (n >= NearCopy::kMin && n <= NearCopy::kMax) {
      NearCopy::get().copy(dst, src, n);
      return;
    }
    constexpr size_t kMinPart = (size_t)512 << 10;
    const size_t parts = std::min<size_t>(workers_.size() + 1, (n + kMinPart - 1) / kMinPart);
    if (parts <= 1) {
      std::memcpy(dst, src, n);
      return;
    }
    const size_t part = (n + parts - 1) / parts;
    Latch latch;
    latch.left = parts - 1;
    {
      std::lock_guard<std::mutex> g(mu_);
      for (size_t p = 1; p < parts; ++p) {
        const size_t off = p * part;
        jobs_.push_back({static_cast<char*>(dst) + off, static_cast<const char*>(src) + off,
                         std::min(part, n - off), &latch});
      }
    }
    cv_.notify_all();
    std::memcpy(dst, src, std::min(part, n));
    std::unique_lock<std::mutex> lk(latch.mu);
    latch.cv.wait(lk, [&] { return latch.left == 0; });
  }

 private:
  struct Latch {
    std::mutex mu;
    std::condition_variable cv;
    size_t left = 0;
  };
  struct Job {
    char* dst;
    const char* src;
    size_t n;
    Latch* latch;
  };

  CopyPool() {
    const unsigned hw = std::thread::hardware_concurrency();
    const unsigned n = hw > 1 ? std::min(hw, 16u) - 1 : 0;
    for (unsigned i = 0; i < n; ++i) {
      workers_.emplace_back([this] { run(); });
      workers_.back().detach();
    }
  }

  void run() {
    for (;;) {
      Job j;
      {
        std::unique_lock<std::mutex> lk(mu_);
        cv_.wait(lk, [&] { return !jobs_.empty(); });
        j = jobs_.front();
        jobs_.pop_front();
      }
      std::memcpy(j.dst, j.src, j.n);
      std::lock_guard<std::mutex> g(j.latch->mu);
      if (--j.latch->left == 0) j.latch->cv.notify_all();
    }
  }

  std::vector<std::thread> workers_;
  std::mutex mu_;
  std::condition_variable cv_;
  std::deque<Job> jobs_;
};

// Pinned staging slots of one host thread on one device: each slot's event
// marks the end of the last copy that used it.
class Staging {
 public:
  static constexpr int kSlots = 4;
  static constexpr size_t kSlotBytes = (size_t)64 << 20;

  static Staging& get() {
    static thread_local std::map<int, Staging> per_device;
    int dev = 0;
    CMM_CUDA(cudaGetDevice(&dev));
    return per_device[dev];
  }

  Staging() = default;
  Staging(const Staging&) = delete;
  Staging& operator=(const Staging&) = delete;
  ~Staging() {
    for (int i = 0; i < kSlots; ++i) {
      if (ev_[i]) cudaEventDestroy(ev_[i]);
      if (buf_[i]) cudaFreeHost(buf_[i]);
    }
  }

  // slot i, free for host access (its last copy has completed)
  char* slot(int i) {
    if (!buf_[i]) {
      CMM_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&buf_[i]), kSlotBytes, cudaHostAllocDefault));
      CMM_CUDA(cudaEventCreateWithFlags(&ev_[i], cudaEventDisableTiming));
    } else {
      CMM_CUDA(cudaEventSynchronize(ev_[i]));
    }
    return buf_[i];
  }
  cudaEvent_t event(int i) { return ev_[i]; }
  int next() {
    const int i = next_;
    next_ = (next_ + 1) % kSlots;
    return i;
  }

 private:
  char* buf_[kSlots] = {};
  cudaEvent_t ev_[kSlots] = {};
  int next_ = 0;
};

bool pageable(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

}  // namespace

void host_to_device(void* dst, const void* src, size_t bytes, cudaStream_t cs) {
  if (bytes == 0) return;
  if (!pageable(src)) {
    CMM_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, cs));
    return;
  }
  Staging& st = Staging::get();
  for (size_t off = 0; off < bytes; off += Staging::kSlotBytes) {
    const size_t n = std::min(Staging::kSlotBytes, bytes - off);
    const int i = st.next();
    char* s = st.slot(i);
    CopyPool::get().copy(s, static_cast<const char*>(src) + off, n);
    CMM_CUDA(cudaMemcpyAsync(static_cast<char*>(dst) + off, s, n, cudaMemcpyHostToDevice, cs));
    CMM_CUDA(cudaEventRecord(st.event(i), cs));
  }
}

void device_to_host(void* dst, const void* src, size_t bytes, cudaStream_t cs) {
  if (bytes == 0) return;
  if (!pageable(dst)) {
    CMM_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, cs));
    return;
  }
  // the DMA of up to kSlots pieces is in flight while the host drains the
  // oldest one
  Staging& st = Staging::get();
  struct Piece {
    size_t off, n;
    int slot;
    char* buf;
  };
  std::deque<Piece> inflight;
  auto drain = [&] {
    const Piece p = inflight.front();
    inflight.pop_front();
    CMM_CUDA(cudaEventSynchronize(st.event(p.slot)));
    CopyPool::get().copy(static_cast<char*>(dst) + p.off, p.buf, p.n);
  };
  for (size_t off = 0; off < bytes; off += Staging::kSlotBytes) {
    if ((int)inflight.size() == Staging::kSlots) drain();
    const size_t n = std::min(Staging::kSlotBytes, bytes - off);
    const int i = st.next();
    char* s = st.slot(i);
    CMM_CUDA(cudaMemcpyAsync(s, static_cast<const char*>(src) + off, n, cudaMemcpyDeviceToHost, cs));
    CMM_CUDA(cudaEventRecord(st.event(i), cs));
    inflight.push_back({off, n, i, s});
  }
  while (!inflight.empty()) drain();
}

}  // namespace cmm
