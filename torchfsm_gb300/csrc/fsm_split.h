// The order in which the parts of a split batch are enqueued on their streams, host C++ only.
#pragma once

namespace fsm {

// The parts advance step by step; every `ring` steps each part waits for the part before it (a
// ring), so that none runs far ahead and leaves the others alone at the end. Ops (0: done):
//   fork()       marks the caller's stream         begin(h)    part h's stream waits for the mark
//   prime(h)     part h's work before its steps    step(h, k)  part h's work of step k
//   record(h)    marks part h's stream             wait(h, g)  part h waits for part g's mark
//   join(h)      the caller's stream waits for part h's mark
//   finish(h)    the caller's stream waits for all that part h has enqueued, or the host does
// Whatever fails, the caller's stream waits for all that has been enqueued: the caller gives its
// buffers back on that stream.
template <class Ops>
int run_parts(Ops& ops, int parts, int steps, int ring) {
  int begun = 0;
  int rc = ops.fork();
  for (int h = 0; h < parts && !rc; ++h) {
    if ((rc = ops.begin(h))) break;
    ++begun;
    rc = ops.prime(h);
    if (!rc) rc = ops.record(h);
  }
  for (int k = 0; k < steps && !rc; ++k) {
    for (int h = 0; h < parts && !rc; ++h) {
      if (k % ring == 0) rc = ops.wait(h, (h + parts - 1) % parts);
      if (!rc) rc = ops.step(h, k);
    }
    if ((k + 1) % ring != 0 && k + 1 < steps) continue;
    for (int h = 0; h < parts && !rc; ++h) rc = ops.record(h);
  }
  for (int h = 0; h < parts && !rc; ++h) rc = ops.join(h);
  if (rc)
    for (int h = 0; h < begun; ++h) ops.finish(h);
  return rc;
}

}  // namespace fsm
