// The multi-plan column launch refuses what its kernels do not hold, before any launch: stages of other
// schemes than SETDRK4 (they need shared memory that this launch does not reserve) and mixed launches.
#include <cstdio>
#include <cstring>

#include "fsm_internal.cuh"

int main() {
  int failures = 0;
  auto refused = [&](const char* what, int stage0, int integ0, int stage1, int integ1) {
    fsm::PlaneMulti m;
    memset(&m, 0, sizeof(m));
    m.count = 2;
    for (int j = 0; j < 2; ++j) {
      m.n[j] = 64;
      m.a[j].B = 1;
      m.a[j].stage = j ? stage1 : stage0;
      m.a[j].integ = j ? integ1 : integ0;
    }
    if (fsm::launch_plane_col_multi(m, FSM_NL_CONVECTION, nullptr) != FSM_ERR_UNSUPPORTED) {
      std::printf("not refused: %s\n", what);
      ++failures;
    }
  };
  refused("a stage of SETDRK3", 0, FSM_SETDRK3, 0, FSM_SETDRK3);
  refused("a Runge-Kutta stage beside SETDRK4", 1, FSM_SETDRK4, 1, FSM_RK4);
  refused("a priming entry and a stage", -1, FSM_SETDRK4, 0, FSM_SETDRK4);
  refused("a stage and a priming entry", 0, FSM_SETDRK4, -1, FSM_SETDRK4);
  refused("a stage beyond the scheme's", 4, FSM_SETDRK4, 4, FSM_SETDRK4);
  if (failures == 0) std::printf("ok\n");
  return failures;
}
