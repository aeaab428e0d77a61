// Host memory copied by several threads (host_copy.cu). No CUDA in here: the threads' protocol is also compiled by itself,
// under the thread sanitizer.
#pragma once
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

namespace cgtb {

constexpr size_t kChunk = 256 << 10;

// Into pinned memory that the GPU reads next: stores that bypass the caches. Lines left modified in several cores' caches
// are fetched from there by every read over PCIe (6.1 MB written by four threads: 650 us until the copy engine is
// done, 185 us with these stores).
inline void stream_to_pinned(char* dst, const char* src, size_t n) {
  size_t i = 0;
#if defined(__SSE2__)
  if (((uintptr_t)dst & 15) == 0) {
    for (; i + 64 <= n; i += 64) {
      _mm_prefetch(src + i + 1024, _MM_HINT_NTA);
      const __m128i a = _mm_loadu_si128((const __m128i*)(src + i)), b = _mm_loadu_si128((const __m128i*)(src + i + 16)),
                    c = _mm_loadu_si128((const __m128i*)(src + i + 32)), d = _mm_loadu_si128((const __m128i*)(src + i + 48));
      _mm_stream_si128((__m128i*)(dst + i), a);
      _mm_stream_si128((__m128i*)(dst + i + 16), b);
      _mm_stream_si128((__m128i*)(dst + i + 32), c);
      _mm_stream_si128((__m128i*)(dst + i + 48), d);
    }
    _mm_sfence();
  }
#endif
  memcpy(dst + i, src + i, n - i);
}

// Three helper threads, asleep between copies. A copy is cut into chunks that the caller and whoever is awake take one
// after the other, so a helper that needs long to wake (a halted virtual CPU: tens of microseconds) delays nothing. A
// caller that finds the helpers busy with another thread's copy copies alone.
class CopyThreads {
 public:
  static constexpr int kHelpers = 3;
  ~CopyThreads() {
    {
      std::lock_guard<std::mutex> lk(mu_);
      stop_ = true;
    }
    cv_.notify_all();
    for (auto& t : threads_) t.join();
  }
  // in_order(first byte, end): called by the copying thread for finished stretches, front to back
  template <typename F>
  void copy(char* dst, const char* src, size_t n, bool to_gpu, F in_order) {
    std::unique_lock<std::mutex> owner(owner_, std::try_to_lock);
    const size_t chunks = (n + kChunk - 1) / kChunk;
    if (!owner.owns_lock() || chunks < 4 || !prepare(chunks)) {
      for (size_t c = 0; c < chunks; ++c) {
        const size_t at = c * kChunk, end = std::min(n, at + kChunk);
        memcpy(dst + at, src + at, end - at);  // alone: a thread's streaming stores are slower than its memcpy
        in_order(at, end);
      }
      return;
    }
    for (size_t c = 0; c < chunks; ++c) done_[c].store(0, std::memory_order_relaxed);
    to_gpu_ = to_gpu;   // the job's fields are the owner's to write, and only while no helper is at work
    dst_ = dst;
    src_ = src;
    bytes_ = n;
    chunks_ = chunks;
    next_.store(0, std::memory_order_relaxed);
    {
      std::lock_guard<std::mutex> lk(mu_);
      open_ = true;
      ++generation_;
    }
    cv_.notify_all();
    size_t issued = 0;
    while (issued < chunks) {
      one_chunk();
      size_t ready = issued;
      while (ready < chunks && done_[ready].load(std::memory_order_acquire)) ++ready;
      if (ready > issued) {
        in_order(issued * kChunk, std::min(n, ready * kChunk));
        issued = ready;
      }
    }
    std::unique_lock<std::mutex> lk(mu_);
    open_ = false;
    idle_.wait(lk, [&] { return active_ == 0; });
  }

 private:
  // The helpers and a flag per chunk. A process at its limit of threads or memory gets none: false, and the caller copies
  // alone (an exception must not leave through the C interface). It is tried again by the next copy.
  bool prepare(size_t chunks) {
    try {
      if (done_.size() < chunks) done_ = std::vector<std::atomic<char>>(chunks);
      threads_.reserve(kHelpers);
      while (threads_.size() < kHelpers) threads_.emplace_back([this] { work(); });
    } catch (const std::exception&) {
    }
    return done_.size() >= chunks && !threads_.empty();
  }
  bool one_chunk() {
    const size_t c = next_.fetch_add(1, std::memory_order_relaxed);
    if (c >= chunks_) return false;
    const size_t at = c * kChunk, end = std::min(bytes_, at + kChunk);
    if (to_gpu_) stream_to_pinned(dst_ + at, src_ + at, end - at);
    else memcpy(dst_ + at, src_ + at, end - at);
    done_[c].store(1, std::memory_order_release);
    return true;
  }
  void work() {
    long seen = 0;
    std::unique_lock<std::mutex> lk(mu_);
    for (;;) {
      cv_.wait(lk, [&] { return stop_ || (open_ && generation_ != seen); });
      if (stop_) return;
      seen = generation_;
      ++active_;
      lk.unlock();
      while (one_chunk()) {}
      lk.lock();
      if (--active_ == 0) idle_.notify_one();
    }
  }
  std::mutex owner_, mu_;
  std::condition_variable cv_, idle_;
  std::vector<std::thread> threads_;
  std::vector<std::atomic<char>> done_;
  std::atomic<size_t> next_{0};
  long generation_ = 0;
  int active_ = 0;
  bool stop_ = false, open_ = false, to_gpu_ = false;
  char* dst_ = nullptr;
  const char* src_ = nullptr;
  size_t bytes_ = 0, chunks_ = 0;
};

}  // namespace cgtb
