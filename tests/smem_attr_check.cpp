// The shared-memory limits of kernels under concurrent callers (fsm_smem_attr.h), with a stand-in for
// the attribute call: the last size set is the one in force.
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <mutex>
#include <thread>

#include "fsm_smem_attr.h"

namespace {

int failures = 0;
void expect(bool ok, const char* what) {
  if (!ok) {
    std::printf("%s\n", what);
    ++failures;
  }
}

// A smaller raise that is inside its attribute call when a larger one begins.
void overlapping() {
  fsm::SmemAttributes attrs;
  int kernel = 0;
  std::atomic<size_t> in_force{0};
  std::mutex m;
  std::condition_variable cv;
  bool small_entered = false, large_done = false;
  std::thread small([&] {
    attrs.raise(&kernel, 0, 70000, [&] {
      std::unique_lock<std::mutex> l(m);
      small_entered = true;
      cv.notify_all();
      cv.wait_for(l, std::chrono::milliseconds(300), [&] { return large_done; });
      in_force = 70000;
      return 0;
    });
  });
  {
    std::unique_lock<std::mutex> l(m);
    cv.wait(l, [&] { return small_entered; });
  }
  attrs.raise(&kernel, 0, 100000, [&] {
    in_force = 100000;
    return 0;
  });
  {
    std::lock_guard<std::mutex> l(m);
    large_done = true;
  }
  cv.notify_all();
  small.join();
  attrs.raise(&kernel, 0, 100000, [&] {
    in_force = 100000;
    return 0;
  });
  expect(in_force >= 100000, "the larger limit is not in force after both calls");
}

void sequential() {
  fsm::SmemAttributes attrs;
  int a = 0, b = 0, calls = 0;
  auto set = [&] {
    ++calls;
    return 0;
  };
  attrs.raise(&a, 0, 60000, set);
  attrs.raise(&a, 0, 60000, set);
  attrs.raise(&a, 0, 50000, set);
  expect(calls == 1, "a limit already in force was set again");
  attrs.raise(&a, 0, 80000, set);
  attrs.raise(&a, 1, 60000, set);
  attrs.raise(&b, 0, 60000, set);
  expect(calls == 4, "a larger size, another device or another kernel was not set");
  expect(attrs.raise(&b, 0, 90000, [] { return 7; }) == 7, "a failure is not returned");
  attrs.raise(&b, 0, 90000, set);
  expect(calls == 5, "a failed call was taken as done");
}

}  // namespace

int main() {
  overlapping();
  sequential();
  if (failures == 0) std::printf("ok\n");
  return failures;
}
