// Work done once for each key on each device of the process (no CUDA here, so
// that it can be tested on the host).
#pragma once

#include <mutex>
#include <set>
#include <utility>

namespace fpls {

// run(key, device, f) calls f the first time the pair comes up and returns
// after it has run, on whichever thread. An f that throws leaves the pair to
// the next caller.
class OncePerDevice {
 public:
  template <class F>
  void run(const void* key, int device, F&& f) {
    std::lock_guard<std::mutex> lock(mu_);
    if (done_.count({key, device})) return;
    f();
    done_.insert({key, device});
  }

 private:
  std::mutex mu_;
  std::set<std::pair<const void*, int>> done_;
};

}  // namespace fpls
