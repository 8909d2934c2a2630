// host_pages.h -- pages of host result arrays.
#pragma once

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstddef>
#include <exception>
#include <thread>
#include <utility>
#include <vector>

namespace fapk {

// Brings the pages of pageable host results in while the GPU works and while the
// array before them is copied.  A result array is usually fresh memory, and the
// copy into it would take a page fault every page on one thread: 184 MB in 6.5 to
// 8.5 ms, 1.0 to 2.5 ms when the pages are there; three threads bring them in in
// 2.4 ms (64 KB pages; one 5.4, two 3.1, four 2.2, six 5.4).  The contents stay
// as they are, and a range or a kernel that refuses is left to the copy.
class HostPages {
 public:
  // Returns the number of pieces so far, for wait().
  size_t add(void *p, size_t bytes) {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    const size_t at = reinterpret_cast<size_t>(p);
    const size_t lo = (at + page - 1) / page * page, hi = (at + bytes) / page * page;
    const size_t step = (kPiece + page - 1) / page * page;
    for (size_t a = lo; a < hi; a += step) pieces_.push_back({a, std::min(step, hi - a)});
    return pieces_.size();
  }
  void start() {
    try {
      for (size_t i = 0; i < std::min<size_t>(kThreads, pieces_.size() / 2); i++) threads_.emplace_back([this] { run(); });
    } catch (const std::exception &) {  // fewer threads, or none
    }
  }
  // Until about the first `n` pieces are in: they are taken in order, but a thread
  // may still hold one of them (the copy then faults its pages in).
  void wait(size_t n) {
    if (n >= pieces_.size()) return join();
    while (!threads_.empty() && next_.load() < std::min(n + threads_.size(), pieces_.size()))
      std::this_thread::sleep_for(std::chrono::microseconds(20));
  }
  void join() {
    for (std::thread &t : threads_) t.join();
    threads_.clear();
  }
  // A solve that failed leaves the rest of the pages alone: a few pieces are
  // finished, not a result array of any size.
  ~HostPages() {
    next_.store(pieces_.size() + kThreads);
    join();
  }

 private:
  static constexpr size_t kPiece = (size_t)4 << 20, kThreads = 3;
  void run() {
#ifdef MADV_POPULATE_WRITE
    for (size_t i; (i = next_.fetch_add(1)) < pieces_.size();)
      if (madvise(reinterpret_cast<void *>(pieces_[i].first), pieces_[i].second, MADV_POPULATE_WRITE) != 0) break;
#endif
    next_.store(pieces_.size() + kThreads);  // (nothing left to take, or refused)
  }
  std::vector<std::pair<size_t, size_t>> pieces_;
  std::vector<std::thread> threads_;
  std::atomic<size_t> next_{0};
};

}  // namespace fapk
