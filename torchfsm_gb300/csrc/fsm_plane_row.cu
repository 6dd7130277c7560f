// The 2D row pass (16..512 points per axis): the kernels of one plan and their launchers. The device
// body is in fsm_plane_reg.cuh.
#include "fsm_plane_reg.cuh"

namespace fsm {

template <int NY, int KIND, int HK>
__global__ void __launch_bounds__(256, 2) k_plane_row_r(StepArgs a) {
  plane_row_body<NY, KIND, HK>(a, blockIdx.x, blockIdx.y);
}

template <int NY, int KIND, int HK>
static int launch_row_r_hk(int nx, const StepArgs& a, cudaStream_t st) {
  using Cfg = RowCfgR<NY>;
  const int groups_needed = nx / 2;
  int threads = groups_needed * Cfg::T;
  if (threads > 256) threads = 256;
  const int groups = threads / Cfg::T;
  const size_t smem = (size_t)(NY + groups * Cfg::SCR) * sizeof(float2);
  int rc = prep_smem(k_plane_row_r<NY, KIND, HK>, smem);
  if (rc) return rc;
  dim3 grid(groups_needed / groups, a.B);
  return launch_pdl(a.pdl, k_plane_row_r<NY, KIND, HK>, grid, threads, smem, st, "k_plane_row_r", a);
}

// The 2/3 rule's stored prefix (NY/3 + 1 columns) or every column.
template <int NY, int KIND>
static int launch_row_r(int nx, const StepArgs& a, cudaStream_t st) {
  if (a.hk == NY / 3 + 1) return launch_row_r_hk<NY, KIND, NY / 3 + 1>(nx, a, st);
  if (a.hk != NY / 2 + 1) return set_error(FSM_ERR_INVALID, "row pass: unexpected stored column count");
  return launch_row_r_hk<NY, KIND, NY / 2 + 1>(nx, a, st);
}

template <int KIND>
static int row_r_dispatch(int nx, int ny, const StepArgs& a, cudaStream_t st) {
  switch (ny) {
    case 16: return launch_row_r<16, KIND>(nx, a, st);
    case 32: return launch_row_r<32, KIND>(nx, a, st);
    case 64: return launch_row_r<64, KIND>(nx, a, st);
    case 128: return launch_row_r<128, KIND>(nx, a, st);
    case 256: return launch_row_r<256, KIND>(nx, a, st);
    case 512: return launch_row_r<512, KIND>(nx, a, st);
  }
  return set_error(FSM_ERR_UNSUPPORTED, "plane pass: unsupported size or nonlinear term");
}

int launch_plane_row(const FsmPlan* p, const StepArgs& a, cudaStream_t st) {
  switch (p->nl) {
    case FSM_NL_VORTICITY: return row_r_dispatch<FSM_NL_VORTICITY>(p->n[0], p->n[1], a, st);
    case FSM_NL_CONVECTION:
    case FSM_NL_LERAY: return row_r_dispatch<FSM_NL_CONVECTION>(p->n[0], p->n[1], a, st);
    case FSM_NL_KS: return row_r_dispatch<FSM_NL_KS>(p->n[0], p->n[1], a, st);
  }
  return set_error(FSM_ERR_UNSUPPORTED, "plane pass: unsupported size or nonlinear term");
}

}  // namespace fsm
