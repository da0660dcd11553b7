// Host blocks lent to calls. Plain C++ (no CUDA header).
#pragma once

#include <mutex>
#include <vector>

namespace dlp {

// Blocks of T that calls of any thread borrow and give back: as many are allocated as were ever borrowed at once,
// however many threads come and go.
template <class T>
class BlockPool {
 public:
  // A free block, else alloc()'s (NULL: none, and nothing to give back).
  template <class Alloc>
  T *borrow(Alloc alloc) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      if (!free_.empty()) {
        T *p = free_.back();
        free_.pop_back();
        return p;
      }
    }
    return alloc();
  }
  void give(T *p) noexcept {
    if (!p) return;
    try {
      std::lock_guard<std::mutex> lk(mu_);
      free_.push_back(p);
    } catch (...) {  // no room for the pointer: the block is not lent again
    }
  }

 private:
  std::mutex mu_;
  std::vector<T *> free_;
};

}  // namespace dlp
