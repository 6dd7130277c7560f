// The resident 2D kernels of the LERAY term (fsm_resident.cuh).
#include "fsm_resident.cuh"

namespace fsm {
ResKernel resident_leray(int nx, int ny) { return resident_kind<FSM_NL_LERAY>(nx, ny); }
}  // namespace fsm
