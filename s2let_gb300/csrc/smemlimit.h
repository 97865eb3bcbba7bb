// Shared-memory attributes of kernels whose launches differ in size (host code).
#pragma once

#include <cstddef>
#include <map>
#include <mutex>

namespace s2g {

// The attributes of a kernel belong to the process, and other threads launch it too:
// the limit on dynamic shared memory is only ever raised, since lowering it between
// another thread's preparation and its launch would make that launch fail.  The
// carveout is a hint and follows the last size asked for.
class SharedMemoryLimits {
 public:
  // set_limit(bytes) and set_carveout(percent) set the kernel's attributes
  template <class L, class C>
  void prepare(const void *kernel, size_t bytes, int percent, L &&set_limit, C &&set_carveout) {
    std::lock_guard<std::mutex> lk(mu_);
    State &s = state_[kernel];
    if (bytes > s.limit) {
      set_limit(bytes);
      s.limit = bytes;
    }
    if (percent != s.percent) {
      set_carveout(percent);
      s.percent = percent;
    }
  }

 private:
  struct State {
    size_t limit = 48 * 1024;  // what a kernel may use without asking
    int percent = -1;
  };
  std::mutex mu_;
  std::map<const void *, State> state_;
};

}  // namespace s2g
