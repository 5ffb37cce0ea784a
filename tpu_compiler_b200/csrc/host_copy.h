// Copies between the caller's pageable arrays and pinned buffers, on several host threads.
//
// setTensor takes ordinary host memory. The driver's own path for that copies on one thread (16-18 GB/s measured) and
// finishes the whole copy before the conversion kernel may start. Here the caller's thread and up to three helpers copy
// small blocks, and each piece is handed to the device as soon as its blocks are there.
//
// One set of helper threads per process, started at the first copy that is large enough, asleep between copies (after a
// short spin). When another thread is using them, a caller copies alone. The helpers never touch CUDA.
#pragma once
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <functional>
#include <mutex>
#include <thread>

#include <unistd.h>
#if defined(__x86_64__)
#include <emmintrin.h>
#endif

namespace tpucb {

// memcpy into a 16-byte aligned pinned buffer that a device copy reads next, past the caches: the link reads lines that
// another core holds modified at 20 GB/s, lines that lie in memory at 50.
inline void stream_copy(void *dst, const void *src, size_t bytes) {
#if defined(__x86_64__)
  uint8_t *d = (uint8_t *)dst;
  const uint8_t *s = (const uint8_t *)src;
  size_t i = 0;
  for (; i + 64 <= bytes; i += 64) {
    const __m128i a = _mm_loadu_si128((const __m128i *)(s + i)), b = _mm_loadu_si128((const __m128i *)(s + i + 16));
    const __m128i c = _mm_loadu_si128((const __m128i *)(s + i + 32)), e = _mm_loadu_si128((const __m128i *)(s + i + 48));
    _mm_stream_si128((__m128i *)(d + i), a);
    _mm_stream_si128((__m128i *)(d + i + 16), b);
    _mm_stream_si128((__m128i *)(d + i + 32), c);
    _mm_stream_si128((__m128i *)(d + i + 48), e);
  }
  if (i < bytes) std::memcpy(d + i, s + i, bytes - i);
  _mm_sfence();
#else
  std::memcpy(dst, src, bytes);
#endif
}

class CopyHelpers {
public:
  // Runs block(i) for every i in [0, n), each exactly once, on this thread and the helpers; after_block(), on this thread
  // only, follows each of its blocks and is called until it returns true once all blocks are taken (it sees what has
  // finished through the caller's own counters).
  static void run(int n, bool parallel, const std::function<void(int)> &block, const std::function<bool()> &after_block) {
    CopyHelpers *h = parallel ? instance() : nullptr;
    std::unique_lock<std::mutex> use;
    if (h) {
      use = std::unique_lock<std::mutex>(h->use_, std::try_to_lock);
      if (!use.owns_lock()) h = nullptr;
    }
    if (!h) {
      for (int i = 0; i < n; ++i) {
        block(i);
        after_block();
      }
      while (!after_block()) {
      }
      return;
    }
    h->block_ = &block;
    h->n_ = n;
    h->next_.store(0);
    h->open_.store(true);
    h->job_.fetch_add(1);
    if (h->asleep_.load() > 0) { // (the lock: a helper that has just looked at job_ is by now inside its wait)
      { std::lock_guard<std::mutex> lock(h->m_); }
      h->cv_.notify_all();
    }
    for (int i; (i = h->next_.fetch_add(1)) < n;) {
      block(i);
      after_block();
    }
    while (!after_block()) pause();
    // No helper enters this job any more, and those inside have found no block left. No mutex here: helpers that are only
    // now being woken would hold it while this thread waits for them (500 us instead of 60 in one call of ten).
    h->open_.store(false);
    while (h->inside_.load() > 0) pause();
  }

private:
  static CopyHelpers *instance() {
    static std::mutex m;
    static CopyHelpers *h = nullptr;
    static pid_t owner = 0;
    std::lock_guard<std::mutex> lock(m);
    if (!h || owner != getpid()) { // the threads do not survive a fork
      h = new CopyHelpers();
      owner = getpid();
    }
    return h;
  }
  CopyHelpers() {
    const unsigned cores = std::thread::hardware_concurrency();
    const int helpers = cores >= 8 ? 3 : (cores >= 4 ? 1 : 0);
    try {
      for (int i = 0; i < helpers; ++i) std::thread([this] { loop(); }).detach();
    } catch (...) { // no more threads to be had: those that run are enough, and none are, too
    }
  }
  static void pause() {
#if defined(__x86_64__)
    _mm_pause();
#endif
  }
  void loop() {
    unsigned seen = 0;
    for (;;) {
      for (int spin = 0; spin < 400 && job_.load() == seen; ++spin) pause();
      if (job_.load() == seen) {
        std::unique_lock<std::mutex> lock(m_);
        asleep_.fetch_add(1);
        cv_.wait(lock, [&] { return job_.load() != seen; });
        asleep_.fetch_sub(1);
      }
      seen = job_.load();
      inside_.fetch_add(1); // before the look at open_: whoever closes the job sees this helper, or it sees the job closed
      if (open_.load()) {
        const std::function<void(int)> &block = *block_;
        const int n = n_;
        for (int i; (i = next_.fetch_add(1)) < n;) block(i);
      }
      inside_.fetch_sub(1);
    }
  }

  std::mutex use_, m_;
  std::condition_variable cv_;
  std::atomic<unsigned> job_{0};
  std::atomic<int> next_{0}, inside_{0}, asleep_{0};
  std::atomic<bool> open_{false};
  const std::function<void(int)> *block_ = nullptr;
  int n_ = 0;
};

} // namespace tpucb
