// The word that a tensor-core kernel sets when one of its bounded waits gives
// up, in host memory that the device writes.  Each owner of launches (a
// backend, a setup level) has a word of its own and reads it after its own
// synchronisation, so that the call which failed reports it, and only that one.
#pragma once
#include <mutex>
#include <vector>

#include "qacode.h"

namespace qf {

// Words in pages of host memory, handed out one by one and taken back: as many
// as there are owners at a time.  `alloc` gives a page of kPage words, `alive`
// says whether a page is still there (a device reset takes it away).
class WaitWords {
 public:
  static constexpr size_t kPage = 1024;
  using Alloc = int* (*)();
  using Alive = bool (*)(const int*);
  WaitWords(Alloc alloc, Alive alive) : alloc_(alloc), alive_(alive) {}
  int* take() {
    std::lock_guard<std::mutex> lock(mu_);
    if (!pages_.empty() && !alive_(pages_.back())) {
      pages_.clear();
      free_.clear();
    }
    if (free_.empty()) {
      pages_.push_back(alloc_());
      for (size_t i = kPage; i-- > 0;) free_.push_back(pages_.back() + i);
    }
    int* p = free_.back();
    free_.pop_back();
    *p = 0;
    return p;
  }
  void put(int* p) {
    std::lock_guard<std::mutex> lock(mu_);
    for (const int* page : pages_)
      if (p >= page && p < page + kPage) {
        free_.push_back(p);
        return;
      }
  }

 private:
  std::mutex mu_;
  Alloc alloc_;
  Alive alive_;
  std::vector<int*> pages_, free_;
};

class WaitFlag {
 public:
  explicit WaitFlag(WaitWords& words) : words_(words) {}
  ~WaitFlag() {
    if (p_) words_.put(p_);
  }
  WaitFlag(const WaitFlag&) = delete;
  WaitFlag& operator=(const WaitFlag&) = delete;
  // The word for a launch; taken at the first one.
  int* word() {
    if (!p_) p_ = words_.take();
    return p_;
  }
  // After the launches' stream has been waited for: fails if a wait gave up
  // since the last check, once.
  void check() {
    if (!p_ || !*static_cast<volatile int*>(p_)) return;
    *p_ = 0;
    fail(QF_E_CUDA, "CUDA: a tensor-core kernel gave up waiting");
  }

 private:
  WaitWords& words_;
  int* p_ = nullptr;
};

}  // namespace qf
