// The dynamic shared-memory limit set for each (kernel, device), host C++ only. Setting the limit
// replaces the one before, so one lock covers look-up, set and record: two threads that raise one
// kernel's limit to different sizes leave the larger one in force.
#pragma once

#include <cstddef>
#include <map>
#include <mutex>
#include <utility>

namespace fsm {

class SmemAttributes {
 public:
  // Have at least `bytes` in force: calls set() (0: done) where less is. Returns set()'s answer, or 0.
  template <class Set>
  int raise(const void* kernel, int device, size_t bytes, Set&& set) {
    std::lock_guard<std::mutex> lock(m_);
    size_t& known = limit_[{kernel, device}];
    if (bytes <= known) return 0;
    const int rc = set();
    if (rc == 0) known = bytes;
    return rc;
  }

 private:
  std::mutex m_;
  std::map<std::pair<const void*, int>, size_t> limit_;
};

}  // namespace fsm
