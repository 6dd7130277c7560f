// The column pass kernels of the LERAY term.
#include "fsm_plane_col.cuh"

namespace fsm {
int launch_col_leray(const FsmPlan* p, const StepArgs& a, cudaStream_t st) {
  if (p->ndim == 3) return col_r_dispatch<FSM_NL_LERAY, 3>(p->n[0], a, st);
  return col_r_dispatch<FSM_NL_LERAY, 2>(p->n[0], a, st);
}
}  // namespace fsm
