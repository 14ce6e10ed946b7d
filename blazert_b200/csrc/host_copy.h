// Copies between ordinary (pageable) host memory and pinned staging on several threads.
#pragma once
#include <atomic>
#include <algorithm>
#include <chrono>
#include <cstddef>
#include <cstring>
#include <thread>
#include <vector>

namespace bzr {

struct HostCopy {
  void *dst;
  const void *src;
  size_t bytes;
};

// A few threads that live as long as the object and share each set of copies by bytes.  One
// thread copies at 5 to 10 GB/s and takes the page faults of a fresh result array one by one;
// the copies of a ray batch's chunks follow each other within microseconds, so an idle thread
// polls, yielding, for a few hundred microseconds before it starts to sleep in between.  A thread
// that cannot be started leaves its share to the others.
class CopyCrew {
 public:
  explicit CopyCrew(size_t threads) {
    try {
      workers_.reserve(threads);
      for (size_t w = 1; w < threads; ++w) workers_.emplace_back([this] { work(); });
    } catch (...) {
    }
  }
  ~CopyCrew() {
    stop_.store(true, std::memory_order_release);
    for (std::thread &t : workers_) t.join();
  }
  CopyCrew(const CopyCrew &) = delete;
  CopyCrew &operator=(const CopyCrew &) = delete;

  // Runs the copies; returns when all are done.
  void run(const HostCopy *copies, size_t n) {
    copies_ = copies;
    n_ = n;
    total_ = 0;
    for (size_t j = 0; j < n; ++j) total_ += copies[j].bytes;
    done_.store(0, std::memory_order_relaxed);
    next_.store(0, std::memory_order_relaxed);
    round_.fetch_add(1, std::memory_order_release);
    pieces();
    // the workers that joined this round still read copies_: wait for each
    while (done_.load(std::memory_order_acquire) < workers_.size()) std::this_thread::yield();
  }

 private:
  static constexpr size_t kPiece = size_t(256) << 10;

  // Takes pieces of the round's bytes, laid end to end, until none is left.
  void pieces() {
    for (;;) {
      const size_t a = next_.fetch_add(kPiece, std::memory_order_relaxed);
      if (a >= total_) return;
      size_t from = a, left = std::min(kPiece, total_ - a);
      for (size_t j = 0; left && j < n_; ++j) {
        if (from >= copies_[j].bytes) {
          from -= copies_[j].bytes;
          continue;
        }
        const size_t m = std::min(left, copies_[j].bytes - from);
        std::memcpy(static_cast<char *>(copies_[j].dst) + from,
                    static_cast<const char *>(copies_[j].src) + from, m);
        left -= m;
        from = 0;
      }
    }
  }
  void work() {
    int idle = 0;
    for (unsigned seen = 0;;) {
      const unsigned r = round_.load(std::memory_order_acquire);
      if (r == seen) {
        if (stop_.load(std::memory_order_acquire)) return;
        if (++idle < 1000)
          std::this_thread::yield();
        else
          std::this_thread::sleep_for(std::chrono::microseconds(20));
        continue;
      }
      idle = 0;
      seen = r;
      pieces();
      done_.fetch_add(1, std::memory_order_release);
    }
  }

  std::vector<std::thread> workers_;
  const HostCopy *copies_ = nullptr;
  size_t n_ = 0, total_ = 0;
  std::atomic<size_t> next_{0}, done_{0};
  std::atomic<unsigned> round_{0};
  std::atomic<bool> stop_{false};
};

}  // namespace bzr
