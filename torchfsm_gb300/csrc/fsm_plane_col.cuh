// Kernels and launchers of the column pass (x pass in 3D), one nonlinear term per translation unit
// (fsm_plane_col_*.cu). The device bodies are in fsm_plane_reg.cuh.
#pragma once

#include "fsm_plane_reg.cuh"

namespace fsm {

// Channel groups of a program: adjacent CTAs of grid.x, so that the coefficient tables that one channel's
// CTA reads from memory are in L2 for the others'.
template <int KIND, int DIM>
constexpr int kGroups = RegKind<KIND, DIM>::C / RegKind<KIND, DIM>::CG;

template <int NX, int KIND, int DIM>
__global__ void __launch_bounds__(256, RegKind<KIND, DIM>::CG == 1 ? 2 : 1) k_axis0_r(StepArgs a) {
  axis0_body<NX, KIND, DIM, false>(a, blockIdx.x / kGroups<KIND, DIM>, blockIdx.y, blockIdx.x % kGroups<KIND, DIM>);
}

template <int NX, int KIND, int DIM, int STG>
__global__ void __launch_bounds__(256, 2) k_axis0_r2(StepArgs a) {
  axis0_body<NX, KIND, DIM, true, STG>(a, blockIdx.x / kGroups<KIND, DIM>, blockIdx.y, blockIdx.x % kGroups<KIND, DIM>);
}

template <int NX, int KIND, int DIM, int STG>
static int launch_axis0_r_mode(const StepArgs& a, cudaStream_t st) {
  using Cfg = ColCfg<NX>;
  // the schemes dispatched at run time pass their points through words of their own
  const bool any = STG < 0 && a.stage >= 0 && a.integ != FSM_SETDRK4 && a.integ != FSM_APPLY;
  const size_t smem = (size_t)(Cfg::WORDS + (any ? RegKind<KIND, DIM>::CG * Cfg::E * 256 : 0)) * sizeof(float2);
  const int64_t inner = a.S / NX;
  dim3 grid((unsigned)((inner + Cfg::W - 1) / Cfg::W) * kGroups<KIND, DIM>, a.B);
  if constexpr (STG >= 0) {
    int rc = prep_smem(k_axis0_r2<NX, KIND, DIM, STG>, smem);
    if (rc) return rc;
    return launch_pdl(a.pdl, k_axis0_r2<NX, KIND, DIM, STG>, grid, 256, smem, st, "k_axis0_r2", a);
  } else {
    int rc = prep_smem(k_axis0_r<NX, KIND, DIM>, smem);
    if (rc) return rc;
    return launch_pdl(a.pdl, k_axis0_r<NX, KIND, DIM>, grid, 256, smem, st, "k_axis0_r", a);
  }
}

template <int NX, int KIND, int DIM>
static int launch_axis0_r(const StepArgs& a, cudaStream_t st) {
  constexpr bool fast = RegKind<KIND, DIM>::CG == 1;
  if constexpr (fast) {
    if (a.integ == FSM_SETDRK4) {
      switch (a.stage) {
        case 0: return launch_axis0_r_mode<NX, KIND, DIM, 0>(a, st);
        case 1: return launch_axis0_r_mode<NX, KIND, DIM, 1>(a, st);
        case 2: return launch_axis0_r_mode<NX, KIND, DIM, 2>(a, st);
        case 3: return launch_axis0_r_mode<NX, KIND, DIM, 3>(a, st);
      }
    }
  }
  return launch_axis0_r_mode<NX, KIND, DIM, -1>(a, st);
}

template <int KIND, int DIM>
int col_r_dispatch(int nx, const StepArgs& a, cudaStream_t st) {
  switch (nx) {
    case 16: return launch_axis0_r<16, KIND, DIM>(a, st);
    case 32: return launch_axis0_r<32, KIND, DIM>(a, st);
    case 64: return launch_axis0_r<64, KIND, DIM>(a, st);
    case 128: return launch_axis0_r<128, KIND, DIM>(a, st);
    case 256: return launch_axis0_r<256, KIND, DIM>(a, st);
    case 512:
      if constexpr (DIM == 2) return launch_axis0_r<512, KIND, DIM>(a, st);
  }
  return set_error(FSM_ERR_UNSUPPORTED, "plane pass: unsupported size or nonlinear term");
}

// 2D and 3D launches of each term.
int launch_col_vorticity(const FsmPlan* p, const StepArgs& a, cudaStream_t st);
int launch_col_convection(const FsmPlan* p, const StepArgs& a, cudaStream_t st);
int launch_col_leray(const FsmPlan* p, const StepArgs& a, cudaStream_t st);
int launch_col_ks(const FsmPlan* p, const StepArgs& a, cudaStream_t st);

}  // namespace fsm
