// host_copy.h -- copies between a caller's pageable arrays and the pinned
// blocks that the device reads and writes.
//
// One core moves some 8 GB/s between pageable memory and a pinned block (page
// faults of fresh result arrays included), a sixth of what the bus takes, so
// large sets of arrays are cut into pieces that the caller's thread and a few
// helper threads copy together.  The helpers belong to the process: they are
// started by the first large copy, never more than kHelpers, and sleep between
// copies.  One copy uses them at a time; a second one made meanwhile by
// another thread is done by that thread alone.
#pragma once

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstddef>
#include <cstring>
#include <memory>
#include <initializer_list>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>
#include <vector>

namespace eplace {

struct CopySpan {
  void *dst;
  const void *src;
  size_t bytes;
};

class HostCopy {
 public:
  static HostCopy &get() {
    static HostCopy *h = new HostCopy();  // never destroyed (its threads live until exit)
    return *h;
  }
  void run(std::initializer_list<CopySpan> spans) {
    size_t total = 0;
    for (const CopySpan &s : spans) total += s.bytes;
    std::unique_lock<std::mutex> one(run_mu_, std::defer_lock);
    std::shared_ptr<Work> w;
    if (total >= kShare && one.try_lock() && start()) {
      try {
        w = std::make_shared<Work>();
        for (const CopySpan &s : spans)
          for (size_t at = 0; at < s.bytes; at += kPiece)
            w->pieces.push_back({static_cast<char *>(s.dst) + at, static_cast<const char *>(s.src) + at,
                                 s.bytes - at < kPiece ? s.bytes - at : kPiece});
      } catch (const std::bad_alloc &) {
        w.reset();
      }
    }
    if (!w) {
      for (const CopySpan &s : spans)
        if (s.bytes) std::memcpy(s.dst, s.src, s.bytes);
      return;
    }
    {
      std::lock_guard<std::mutex> g(mu_);
      work_ = w;
      gen_.fetch_add(1, std::memory_order_release);
    }
    cv_.notify_all();
    help(*w);
    while (w->done.load(std::memory_order_acquire) < w->pieces.size()) std::this_thread::yield();
    std::lock_guard<std::mutex> g(mu_);
    work_.reset();
  }

 private:
  static constexpr int kHelpers = 3;
  static constexpr size_t kShare = 512 << 10;   // smaller sets: waking a helper costs more than it saves
  static constexpr size_t kPiece = 128 << 10;
  struct Work {
    std::vector<CopySpan> pieces;
    std::atomic<size_t> next{0}, done{0};
  };
  static void help(Work &w) {
    for (size_t i; (i = w.next.fetch_add(1, std::memory_order_relaxed)) < w.pieces.size();) {
      std::memcpy(w.pieces[i].dst, w.pieces[i].src, w.pieces[i].bytes);
      w.done.fetch_add(1, std::memory_order_release);
    }
  }
  bool start() {  // run_mu_ held
    if (started_) return helpers_ > 0;
    started_ = true;
    const int spare = (int)std::thread::hardware_concurrency() - 1;
    for (int k = 0; k < kHelpers && k < spare; ++k) {
      try {
        std::thread([this] { loop(); }).detach();
        ++helpers_;
      } catch (const std::system_error &) {
        break;  // fewer helpers, or none
      }
    }
    return helpers_ > 0;
  }
  void loop() {
    uint64_t seen = 0;
    for (;;) {
      // A call makes several copies in a row: look for the next one for a
      // little while before going to sleep.
      const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(50);
      while (gen_.load(std::memory_order_acquire) == seen && std::chrono::steady_clock::now() < until)
        std::this_thread::yield();
      std::shared_ptr<Work> w;
      {
        std::unique_lock<std::mutex> g(mu_);
        cv_.wait(g, [&] { return gen_.load(std::memory_order_relaxed) != seen; });
        seen = gen_.load(std::memory_order_relaxed);
        w = work_;
      }
      if (w) help(*w);
    }
  }
  std::mutex run_mu_, mu_;
  std::condition_variable cv_;
  std::shared_ptr<Work> work_;
  std::atomic<uint64_t> gen_{0};
  bool started_ = false;
  int helpers_ = 0;
};

}  // namespace eplace
