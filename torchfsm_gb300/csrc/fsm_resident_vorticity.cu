// The resident 2D kernels of the VORTICITY term (fsm_resident.cuh).
#include "fsm_resident.cuh"

namespace fsm {
ResKernel resident_vorticity(int nx, int ny) { return resident_kind<FSM_NL_VORTICITY>(nx, ny); }
}  // namespace fsm
