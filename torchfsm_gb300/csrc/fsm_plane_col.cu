// The column pass (2D; the x pass of 3D) by nonlinear term, and the KS batch mean.
#include "fsm_plane_col.cuh"

namespace fsm {

int launch_plane_col(const FsmPlan* p, const StepArgs& a, cudaStream_t st) {
  switch (p->nl) {
    case FSM_NL_VORTICITY: return launch_col_vorticity(p, a, st);
    case FSM_NL_CONVECTION: return launch_col_convection(p, a, st);
    case FSM_NL_LERAY: return launch_col_leray(p, a, st);
    case FSM_NL_KS: return launch_col_ks(p, a, st);
  }
  return set_error(FSM_ERR_UNSUPPORTED, "plane pass: unsupported nonlinear term");
}

// Batch mean of the k = 0 product (KS mean removal): dc = (1/B) sum_b sum_x prod[b][0][x][0..0],
// the products being transformed along every axis but the first.
__global__ void k_ks_mean(StepArgs a, int nx) {
  pdl_wait();
  float acc = 0.f;
  const int total = a.B * nx;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int b = i / nx, x = i % nx;
    acc += a.prod[((int64_t)b * a.n_prod) * a.ms + (int64_t)x * a.wp].x;
  }
  pdl_trigger();
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
  return launch_pdl(a.pdl, k_ks_mean, 1, 256, 0, st, "k_ks_mean", a, p->n[0]);
}

}  // namespace fsm
