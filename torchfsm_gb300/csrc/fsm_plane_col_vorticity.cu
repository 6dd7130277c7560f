// The column pass kernels of the VORTICITY term.
#include "fsm_plane_col.cuh"

namespace fsm {
int launch_col_vorticity(const FsmPlan* p, const StepArgs& a, cudaStream_t st) {
  return col_r_dispatch<FSM_NL_VORTICITY, 2>(p->n[0], a, st);
}
}  // namespace fsm
