// What threads leave behind for the next ones (pure host C++, no CUDA).
//
// A thread owns a resource that is expensive to make and to free: both wait
// for the device and for every other thread that does the same.  Freed with its
// thread, as the slots of the result copies were (1 MB of pinned memory, five
// events, a stream), it made 48 jobs on threads of their own, eight at a time,
// take 95 ms where plain copies took 32 and where resources that are handed on
// take 27.  So
//  * a thread that ends leaves its resource here, and the next that asks has it;
//  * if none lies here, the first of the process is made at once; any other
//    only for a thread that has asked kPatience times, since most threads that
//    run beside others end before one would have paid;
//  * at most kIdle lie here, and none once the last user of the library is gone.
#pragma once

#include <cstddef>
#include <mutex>
#include <vector>

namespace btam {

template <class R> class IdleList {
 public:
  static constexpr int kPatience = 24;
  static constexpr std::size_t kIdle = 8;

  // One of device dev into r, from here or from make(r); asked: the thread's
  // count of attempts.
  template <class Make> bool acquire(int dev, int &asked, R &r, Make make) {
    {
      std::lock_guard<std::mutex> lock(mu_);
      for (std::size_t k = 0; k < idle_.size(); ++k)
        if (idle_[k].device == dev) {
          r = idle_[k];
          idle_.erase(idle_.begin() + (std::ptrdiff_t)k);
          return true;
        }
      if (++asked < kPatience && made_ > 0) return false;
      ++made_;
    }
    if (make(r)) return true;
    std::lock_guard<std::mutex> lock(mu_);
    --made_;
    return false;
  }

  // Leaves r here, or frees it.
  template <class Free> void leave(R &r, Free free) {
    {
      std::lock_guard<std::mutex> lock(mu_);
      if (users_ > 0 && idle_.size() < kIdle) {
        idle_.push_back(r);
        return;
      }
      --made_;
    }
    free(r);
  }

  // A user of the library came (1) or went (-1).
  template <class Free> void users(int by, Free free) {
    std::vector<R> gone;
    {
      std::lock_guard<std::mutex> lock(mu_);
      users_ += by;
      if (users_ == 0) gone.swap(idle_);
      made_ -= (int)gone.size();
    }
    for (R &r : gone) free(r);
  }

 private:
  std::mutex mu_;
  std::vector<R> idle_;
  int made_ = 0, users_ = 0;
};

}  // namespace btam
