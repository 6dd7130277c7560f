// The 2D column pass (16..512 points along x; also the 3D x pass, 16..256) and the KS batch mean: the
// kernels of one plan and their launchers. The device bodies are in fsm_plane_reg.cuh.
#include "fsm_plane_reg.cuh"

namespace fsm {

// channel groups of a program (grid.z)
template <int KIND, int DIM>
constexpr int kGroups = RegKind<KIND, DIM>::C / RegKind<KIND, DIM>::CG;

template <int NX, int KIND, int DIM>
__global__ void __launch_bounds__(256) k_axis0_r(StepArgs a) {
  axis0_body<NX, KIND, DIM, false>(a, blockIdx.x, blockIdx.y, kGroups<KIND, DIM> > 1 ? blockIdx.z : 0);
}

template <int NX, int KIND, int DIM>
__global__ void __launch_bounds__(256, 2) k_axis0_r2(StepArgs a) {
  axis0_body<NX, KIND, DIM, true>(a, blockIdx.x, blockIdx.y, kGroups<KIND, DIM> > 1 ? blockIdx.z : 0);
}

template <int NX, int KIND, int DIM, bool FAST>
static int launch_axis0_r_mode(const StepArgs& a, cudaStream_t st) {
  using Cfg = ColCfg<NX>;
  using K = RegKind<KIND, DIM>;
  const size_t smem = (size_t)(NX + (K::CG + 1) * Cfg::W * Cfg::P) * sizeof(float2);
  const int64_t inner = a.S / NX;
  dim3 grid((unsigned)((inner + Cfg::W - 1) / Cfg::W), a.B, kGroups<KIND, DIM>);
  if constexpr (FAST) {
    int rc = prep_smem(k_axis0_r2<NX, KIND, DIM>, smem);
    if (rc) return rc;
    k_axis0_r2<NX, KIND, DIM><<<grid, 256, smem, st>>>(a);
    return cuda_check(cudaGetLastError(), "k_axis0_r2");
  } else {
    int rc = prep_smem(k_axis0_r<NX, KIND, DIM>, smem);
    if (rc) return rc;
    k_axis0_r<NX, KIND, DIM><<<grid, 256, smem, st>>>(a);
    return cuda_check(cudaGetLastError(), "k_axis0_r");
  }
}

template <int NX, int KIND, int DIM>
static int launch_axis0_r(const StepArgs& a, cudaStream_t st) {
  // the hoisted update for vorticity and convection (KS keeps the generic kernel: its hoisted
  // instance does not fit two CTAs' registers per SM)
  constexpr bool fast = RegKind<KIND, DIM>::CG == 1 && KIND != FSM_NL_KS;
  if (fast && a.integ == FSM_SETDRK4 && a.stage >= 0) return launch_axis0_r_mode<NX, KIND, DIM, fast>(a, st);
  return launch_axis0_r_mode<NX, KIND, DIM, false>(a, st);
}

template <int KIND, int DIM>
static int col_r_dispatch(int nx, const StepArgs& a, cudaStream_t st) {
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

int launch_plane_col(const FsmPlan* p, const StepArgs& a, cudaStream_t st) {
  if (p->ndim == 3) {
    switch (p->nl) {
      case FSM_NL_CONVECTION: return col_r_dispatch<FSM_NL_CONVECTION, 3>(p->n[0], a, st);
      case FSM_NL_LERAY: return col_r_dispatch<FSM_NL_LERAY, 3>(p->n[0], a, st);
      case FSM_NL_KS: return col_r_dispatch<FSM_NL_KS, 3>(p->n[0], a, st);
    }
    return set_error(FSM_ERR_UNSUPPORTED, "plane pass: unsupported size or nonlinear term");
  }
  switch (p->nl) {
    case FSM_NL_VORTICITY: return col_r_dispatch<FSM_NL_VORTICITY, 2>(p->n[0], a, st);
    case FSM_NL_CONVECTION: return col_r_dispatch<FSM_NL_CONVECTION, 2>(p->n[0], a, st);
    case FSM_NL_LERAY: return col_r_dispatch<FSM_NL_LERAY, 2>(p->n[0], a, st);
    case FSM_NL_KS: return col_r_dispatch<FSM_NL_KS, 2>(p->n[0], a, st);
  }
  return set_error(FSM_ERR_UNSUPPORTED, "plane pass: unsupported size or nonlinear term");
}

// Batch mean of the k = 0 product (KS mean removal): dc = (1/B) sum_b sum_x prod[b][0][x][0..0],
// the products being transformed along every axis but the first.
__global__ void k_ks_mean(StepArgs a, int nx) {
  float acc = 0.f;
  const int total = a.B * nx;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int b = i / nx, x = i % nx;
    acc += a.prod[((int64_t)b * a.n_prod) * a.ms + (int64_t)x * a.wp].x;
  }
  __shared__ float red[256];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) a.dc[0] = make_float2(red[0] / (float)a.B, 0.f);
}

int launch_ks_mean(const FsmPlan* p, const StepArgs& a, cudaStream_t st) {
  k_ks_mean<<<1, 256, 0, st>>>(a, p->n[0]);
  return cuda_check(cudaGetLastError(), "k_ks_mean");
}

}  // namespace fsm
