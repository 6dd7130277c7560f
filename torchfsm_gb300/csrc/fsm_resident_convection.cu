// The resident 2D kernels of the CONVECTION term (fsm_resident.cuh).
#include "fsm_resident.cuh"

namespace fsm {
ResKernel resident_convection(int nx, int ny) { return resident_kind<FSM_NL_CONVECTION>(nx, ny); }
}  // namespace fsm
