// Host side of the host-pointer calls: copies between pageable arrays and pinned buffers.
//
// What bounds a host-pointer call is the PCIe link (54 GB/s measured each way) and what feeds it.
// Two measured facts decide the shape of this code (B200 box, 16 cores):
//  * A DMA transfer that finds its lines in the caches of several cores crawls: 4 MB that eight
//    threads had just memcpy'd into the pinned buffer went to the device in 450-700 us instead of
//    82, and 4 MB coming back into lines that eight threads had read the last time took 320-450.
//    So the copy INTO a pinned buffer uses streaming stores (the lines end up in memory, the
//    transfer runs at 83 us per 4 MB), and the copy OUT of one evicts the lines it has read.
//  * Waking a sleeping thread costs tens of microseconds, as much as copying a megabyte.  The
//    calling thread starts on the first piece at once, the workers spin for a moment after a job
//    before they sleep, and pieces are handed out one by one so that nobody waits for a late one.
// The streaming and evicting copies are x86 code, chosen by what the processor has; others copy with memcpy.
#pragma once
#if defined(__x86_64__)
#include <immintrin.h>
#endif
#include <stdint.h>
#include <string.h>
#include <sys/mman.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace b200 {

#if defined(__x86_64__)
inline void cpu_relax() { _mm_pause(); }

// memcpy with streaming stores.
__attribute__((target("avx2"))) inline void copy_streaming_avx2(char* d, const char* s, size_t n) {
  const size_t head = std::min(n, static_cast<size_t>(-reinterpret_cast<uintptr_t>(d) & 31));
  if (head) memcpy(d, s, head);
  d += head; s += head; n -= head;
  size_t i = 0;
  for (; i + 128 <= n; i += 128) {
    const __m256i a = _mm256_loadu_si256(reinterpret_cast<const __m256i*>(s + i));
    const __m256i b = _mm256_loadu_si256(reinterpret_cast<const __m256i*>(s + i + 32));
    const __m256i c = _mm256_loadu_si256(reinterpret_cast<const __m256i*>(s + i + 64));
    const __m256i e = _mm256_loadu_si256(reinterpret_cast<const __m256i*>(s + i + 96));
    _mm256_stream_si256(reinterpret_cast<__m256i*>(d + i), a);
    _mm256_stream_si256(reinterpret_cast<__m256i*>(d + i + 32), b);
    _mm256_stream_si256(reinterpret_cast<__m256i*>(d + i + 64), c);
    _mm256_stream_si256(reinterpret_cast<__m256i*>(d + i + 96), e);
  }
  if (i < n) memcpy(d + i, s + i, n - i);
  _mm_sfence();
}

// memcpy that leaves the source's lines in no cache; in blocks, so that the eviction finds them
// in the first level.
__attribute__((target("clflushopt"))) inline void copy_and_evict_clflushopt(char* d, const char* s, size_t n) {
  constexpr size_t kBlock = 16384;
  for (size_t off = 0; off < n; off += kBlock) {
    const size_t m = n - off < kBlock ? n - off : kBlock;
    memcpy(d + off, s + off, m);
    for (size_t i = 0; i < m; i += 64) _mm_clflushopt(const_cast<char*>(s + off + i));
  }
  _mm_sfence();
}

inline bool cpu_has_clflushopt() {
  unsigned a = 7, b = 0, c = 0, d = 0;
  __asm__ volatile("cpuid" : "+a"(a), "=b"(b), "+c"(c), "=d"(d));
  return (b >> 23) & 1;
}

inline bool cpu_has_avx2() { return __builtin_cpu_supports("avx2"); }
#else
inline void cpu_relax() {}
inline void copy_streaming_avx2(char* d, const char* s, size_t n) { memcpy(d, s, n); }
inline void copy_and_evict_clflushopt(char* d, const char* s, size_t n) { memcpy(d, s, n); }
inline bool cpu_has_clflushopt() { return false; }
inline bool cpu_has_avx2() { return false; }
#endif

inline void copy_to_pinned(char* d, const char* s, size_t n) {
  static const bool avx2 = cpu_has_avx2();
  if (avx2) copy_streaming_avx2(d, s, n);
  else memcpy(d, s, n);
}
// Out of a pinned buffer; into an array beyond the caches with streaming stores, which do not read the lines they
// overwrite (a call with 616 MB into an array that is used again: 25.7 -> 17.4 ms).
inline void copy_from_pinned(char* d, const char* s, size_t n, bool large) {
  static const bool flush = cpu_has_clflushopt(), avx2 = cpu_has_avx2();
  if (large && avx2) copy_streaming_avx2(d, s, n);
  else if (flush) copy_and_evict_clflushopt(d, s, n);
  else memcpy(d, s, n);
}

// Makes the pages of [d, d + n) present without changing their contents; nothing to do where the last one is.
inline void touch_pages(char* d, size_t n) {
  constexpr uintptr_t kPage = 4096;
  const uintptr_t first = reinterpret_cast<uintptr_t>(d), last = (first + n - 1) & ~(kPage - 1);
  unsigned char present = 0;
  if (mincore(reinterpret_cast<void*>(last), 1, &present) == 0 && (present & 1)) return;
  for (uintptr_t p = first; p < first + n; p = (p & ~(kPage - 1)) + kPage)
    __atomic_fetch_or(reinterpret_cast<char*>(p), 0, __ATOMIC_RELAXED);
}

// A few threads that copy one array together with the caller.  One producer at a time (the
// context's lock).
class CopyPool {
 public:
  // Fewer threads where the system gives no more: the caller alone copies everything, too.
  explicit CopyPool(int nthreads) {
    workers_.reserve(nthreads);
    try {
      for (int i = 1; i < nthreads; ++i) workers_.emplace_back([this] { loop(); });
    } catch (const std::system_error&) {
    }
  }
  ~CopyPool() {
    {
      std::lock_guard<std::mutex> g(mu_);
      stop_.store(true);
    }
    cv_.notify_all();
    for (auto& t : workers_) t.join();
  }
  // Copies `bytes` (to_pinned: into a pinned buffer, else out of one) and returns when done.
  // 128 KB pieces: 32 pages' worth of work per hand-out and 16 pieces in a 2 MB chunk.
  // `large`: the array that a pinned buffer is emptied into is larger than the caches.
  void copy(void* dst, const void* src, size_t bytes, bool to_pinned, bool large = false) {
    run(dst, src, bytes, 128 << 10, to_pinned ? kIn : large ? kOutLarge : kOut);
  }
  // Makes the pages of an array present.  A large numpy array is made of 2 MB pages that the kernel zeroes on their
  // first write, one thread at a time each: copied into in 128 KB pieces, the threads waited for one another's page
  // (a call with a fresh 308 MB result 40 ms, 18 with a page per thread; 64 MB 8.1 and 4.4).  A piece is what lies in one such page.
  void touch(void* dst, size_t bytes) { run(dst, nullptr, bytes, 2 << 20, kTouch); }

 private:
  enum Kind { kIn, kOut, kOutLarge, kTouch };
  void run(void* dst, const void* src, size_t bytes, size_t piece, Kind kind) {
    // the first piece of a touch ends at a boundary of its size
    const size_t lead = kind == kTouch ? reinterpret_cast<uintptr_t>(dst) % piece : 0;
    const uint32_t pieces = static_cast<uint32_t>((bytes + lead + piece - 1) / piece);
    const uint64_t gen = (ticket_.load(std::memory_order_relaxed) >> 32) + 1;
    // nobody takes a piece while the job is being described: a worker takes one by exchanging the
    // ticket it has read, so what it read in between belongs to that ticket's job (the two fences: who
    // has seen any of what follows also sees that the ticket is closed)
    ticket_.store(gen << 32 | 0xffffffffu, std::memory_order_seq_cst);
    std::atomic_thread_fence(std::memory_order_release);
    dst_.store(static_cast<char*>(dst), std::memory_order_relaxed);
    src_.store(static_cast<const char*>(src), std::memory_order_relaxed);
    bytes_.store(bytes, std::memory_order_relaxed);
    pieces_.store(pieces, std::memory_order_relaxed);
    piece_.store(piece, std::memory_order_relaxed);
    lead_.store(lead, std::memory_order_relaxed);
    kind_.store(kind, std::memory_order_relaxed);
    done_.store(0, std::memory_order_relaxed);
    ticket_.store(gen << 32, std::memory_order_seq_cst);
    if (pieces > 1 && sleeping_.load(std::memory_order_seq_cst) > 0) {
      { std::lock_guard<std::mutex> g(mu_); }
      cv_.notify_all();
    }
    work(gen);
    while (done_.load(std::memory_order_acquire) != pieces) cpu_relax();
  }

  void work(uint64_t gen) {
    for (;;) {
      uint64_t t = ticket_.load(std::memory_order_acquire);
      char* d = dst_.load(std::memory_order_relaxed);
      const char* s = src_.load(std::memory_order_relaxed);
      const size_t n = bytes_.load(std::memory_order_relaxed);
      const uint32_t pieces = pieces_.load(std::memory_order_relaxed);
      const size_t piece = piece_.load(std::memory_order_relaxed), lead = lead_.load(std::memory_order_relaxed);
      const Kind kind = kind_.load(std::memory_order_relaxed);
      std::atomic_thread_fence(std::memory_order_acquire);
      const uint32_t i = static_cast<uint32_t>(t);
      if (t >> 32 != gen || i >= pieces) return;
      if (!ticket_.compare_exchange_strong(t, t + 1, std::memory_order_acq_rel)) continue;
      const size_t off = i == 0 ? 0 : i * piece - lead, end = std::min(n, (i + 1) * piece - lead);
      if (kind == kIn) copy_to_pinned(d + off, s + off, end - off);
      else if (kind != kTouch) copy_from_pinned(d + off, s + off, end - off, kind == kOutLarge);
      else touch_pages(d + off, end - off);
      done_.fetch_add(1, std::memory_order_release);
    }
  }
  void loop() {
    uint64_t seen = 0;
    for (;;) {
      // spin for about 50 us (the gap between the chunks of one call), then sleep
      const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(50);
      bool fresh = false;
      do {
        for (int k = 0; k < 32 && !fresh; ++k) {
          fresh = posted() != seen;
          if (!fresh) cpu_relax();
        }
      } while (!fresh && !stop_.load(std::memory_order_relaxed) && std::chrono::steady_clock::now() < until);
      if (!fresh) {
        std::unique_lock<std::mutex> g(mu_);
        sleeping_.fetch_add(1, std::memory_order_seq_cst);
        cv_.wait(g, [&] { return stop_.load() || posted() != seen; });
        sleeping_.fetch_sub(1, std::memory_order_seq_cst);
      }
      if (stop_.load()) return;
      seen = posted();
      work(seen);
    }
  }
  // generation of the last job that is open for work
  uint64_t posted() const {
    const uint64_t t = ticket_.load(std::memory_order_seq_cst);
    return static_cast<uint32_t>(t) == 0xffffffffu ? (t >> 32) - 1 : t >> 32;
  }
  std::vector<std::thread> workers_;
  std::mutex mu_;
  std::condition_variable cv_;
  std::atomic<bool> stop_{false};
  std::atomic<int> sleeping_{0};
  std::atomic<uint64_t> ticket_{0};      // generation << 32 | next piece
  std::atomic<char*> dst_{nullptr};
  std::atomic<const char*> src_{nullptr};
  std::atomic<size_t> bytes_{0};
  std::atomic<uint32_t> pieces_{0}, done_{0};
  std::atomic<size_t> piece_{1}, lead_{0};
  std::atomic<Kind> kind_{kIn};
};

}  // namespace b200
