// The enqueueing of a split batch (fsm_split.h) on stand-in streams: the order of its calls, and, with
// each call failing in turn, that the caller's stream waits for all that the parts have enqueued.
#include <cstdio>
#include <string>
#include <vector>

#include "fsm_split.h"

namespace {

struct Fake {
  int fail_at;  // the call that fails (-1: none)
  int calls = 0;
  std::vector<int> enqueued, marked, waited;  // per part: work items enqueued, marked, waited for by the caller
  std::vector<std::string> log;

  Fake(int parts, int fail) : fail_at(fail), enqueued(parts), marked(parts), waited(parts) {}
  bool failing() { return calls++ == fail_at; }
  int call(const std::string& s) {
    log.push_back(s);
    return failing() ? 1 : 0;
  }
  int work(int h, const std::string& s) {  // two launches, the second one may fail
    log.push_back(s);
    ++enqueued[h];
    if (failing()) return 2;
    ++enqueued[h];
    return 0;
  }
  static std::string id(const char* n, int a) { return std::string(n) + std::to_string(a); }
  int fork() { return call("fork"); }
  int begin(int h) { return call(id("begin", h)); }
  int prime(int h) { return work(h, id("prime", h)); }
  int step(int h, int k) { return work(h, id("step", h) + "." + std::to_string(k)); }
  int record(int h) {
    const int rc = call(id("record", h));
    if (!rc) marked[h] = enqueued[h];
    return rc;
  }
  int wait(int h, int g) { return call(id("wait", h) + "." + std::to_string(g)); }
  int join(int h) {
    const int rc = call(id("join", h));
    if (!rc) waited[h] = marked[h];
    return rc;
  }
  void finish(int h) { waited[h] = enqueued[h]; }
};

}  // namespace

int main() {
  int failures = 0;
  for (int parts : {2, 3, 8})
    for (int steps : {0, 1, 4, 7})
      for (int ring : {1, 4}) {
        Fake ok(parts, -1);
        if (fsm::run_parts(ok, parts, steps, ring) != 0 || ok.waited != ok.enqueued) {
          std::printf("parts %d steps %d ring %d: not joined\n", parts, steps, ring);
          ++failures;
        }
        for (int h = 0; h < parts; ++h)
          if (ok.enqueued[h] != 2 * (1 + steps)) ++failures;
        for (int n = 0; n < ok.calls; ++n) {
          Fake f(parts, n);
          if (fsm::run_parts(f, parts, steps, ring) == 0 || f.waited != f.enqueued) {
            std::printf("parts %d steps %d ring %d: call %d (%s) fails and work is left unjoined\n", parts, steps, ring, n,
                        ok.log[(size_t)n].c_str());
            ++failures;
          }
        }
      }
  // two parts, a wait every second step
  Fake order(2, -1);
  fsm::run_parts(order, 2, 3, 2);
  const char* want =
      "fork begin0 prime0 record0 begin1 prime1 record1 wait0.1 step0.0 wait1.0 step1.0 step0.1 step1.1 record0 record1 "
      "wait0.1 step0.2 wait1.0 step1.2 record0 record1 join0 join1 ";
  std::string got;
  for (const auto& s : order.log) got += s + " ";
  if (got != want) {
    std::printf("order: %s\n", got.c_str());
    ++failures;
  }
  if (failures == 0) std::printf("ok\n");
  return failures;
}
