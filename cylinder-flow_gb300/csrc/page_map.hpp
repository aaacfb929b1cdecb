// Maps the pages of an ordinary host buffer that a copy is about to fill, on several
// cores ahead of the copies (host code only).
#pragma once
#include <sys/mman.h>
#include <unistd.h>
#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <exception>
#include <thread>
#include <vector>

namespace cflbm {

// A dump into fresh memory was bound by the driver's page faults on one core: 226 MB
// took 7.8-9.9 ms, 1.2 ms once the pages are there; mapped by 8 cores just ahead of 32
// MB copies 2.1 ms (4 cores 2.4; MADV_POPULATE_WRITE on 4 / 8 cores, which contend for
// the address space, 3.9 / 6.7; atomics that change no bits 22, as each page is mapped
// for reading first; a pinned bounce buffer emptied by 8 / 12 cores 4.0 / 3.7).  Only
// pages that are not there yet are written to (a zero), and with none missing nothing is
// started: threads that touched every page cost the fields of 256x64x64 (4 x 8 MB) 1.4
// ms in arrays used before.  Ranges with holes and memory that may not be written are for
// the copies to take or to refuse.
class PageMapper {
 public:
  PageMapper() = default;
  PageMapper(const PageMapper &) = delete;
  PageMapper &operator=(const PageMapper &) = delete;
  ~PageMapper() {
    next_ = done_.size();
    for (auto &t : pool_) t.join();
  }

  // Starts to map [p, p + bytes); true when there was something to do.
  bool start(void *p, size_t bytes) {
    p_ = static_cast<char *>(p);
    bytes_ = bytes;
    if (bytes < LEAST || !missing()) return false;
    try {
      done_ = std::vector<std::atomic<char>>(there_.size() * page_ / PIECE + 1);
      const unsigned n = std::max(1u, std::min(8u, std::thread::hardware_concurrency()));
      pool_.reserve(n);
      for (unsigned t = 0; t < n; ++t) pool_.emplace_back([this] { work(); });
    } catch (const std::exception &) {  // no more threads or memory: with what there is
    }
    return !pool_.empty();
  }

  // Returns when the first `upto` bytes are mapped.
  void wait(size_t upto) {
    if (pool_.empty()) return;
    upto += (size_t)(p_ - first_);
    for (; ready_ < done_.size() && ready_ * PIECE < upto; ++ready_)
      while (!done_[ready_].load(std::memory_order_acquire)) std::this_thread::yield();
  }

 private:
  static constexpr size_t LEAST = 8u << 20, PIECE = 2u << 20;

  char *page_of(char *q) const { return q - (uintptr_t)q % page_; }

  // Whether pages of the buffer are missing; there_: which are not.
  bool missing() {
    first_ = page_of(p_);
    const size_t n = (size_t)(p_ + bytes_ - first_);
    try {
      there_.resize((n + page_ - 1) / page_);
    } catch (const std::exception &) {
      return false;
    }
    if (mincore(first_, n, there_.data()) != 0) return false;
    return std::any_of(there_.begin(), there_.end(), [](unsigned char v) { return !(v & 1); });
  }

  void work() {
    const size_t per = std::max<size_t>(1, PIECE / page_);
    int writable = -1;  // a thread's first page tells (which refuses what may not be written)
    for (size_t k; (k = next_.fetch_add(1)) < done_.size();) {
      for (size_t g = k * per; g < std::min((k + 1) * per, there_.size()); ++g) {
        if (there_[g] & 1) continue;
        if (writable < 0) writable = writable_page(first_ + g * page_);
        if (writable) *static_cast<volatile char *>(std::max(p_, first_ + g * page_)) = 0;
      }
      done_[k].store(1, std::memory_order_release);
    }
  }

  static int writable_page(char *page) {
#ifdef MADV_POPULATE_WRITE
    return madvise(page, 1, MADV_POPULATE_WRITE) == 0;
#else
    return 0;  // unknown: the copies map the pages
#endif
  }

  char *p_ = nullptr, *first_ = nullptr;  // the buffer and its first page
  size_t bytes_ = 0, ready_ = 0, page_ = (size_t)sysconf(_SC_PAGESIZE);
  std::vector<unsigned char> there_;
  std::atomic<size_t> next_{0};
  std::vector<std::atomic<char>> done_;
  std::vector<std::thread> pool_;
};

}  // namespace cflbm
