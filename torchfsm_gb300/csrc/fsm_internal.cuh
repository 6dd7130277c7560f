// Internal launchers shared between the torchfsm_gb300 CUDA sources.
#pragma once

#include "fsm_common.cuh"
#include "fsm_smem_attr.h"

namespace fsm {

// Arguments of the fused kernels that advance a batch of half spectra.
struct StepArgs {
  float2* state;              // [B][C][S]
  float2* aux;                // [B][n_aux*C][S] scheme running sums (acc, q)
  float2* mid;                // [B][n_mid][S]  stage fields after the outer-axis inverse transform
  float2* prod;               // [B][n_prod][S] products after the last-axis forward transform
  float2* traj;               // [B][n_frames][C][S]
  int n_frames;
  int slot;                   // frame written at the end of this launch, or -1
  const int32_t* slots;       // device copy of the record slots (single-launch kernels)
  const float2* tab;          // coefficient tables
  int64_t ts;                 // distance between tables
  int lin_batch, lin_ch;
  const float2* src;          // explicit source or null
  int src_batch;
  const float* kx;            // 2 pi f of the first axis
  const float* ky;            // 2 pi f of the last axis
  const float* km;            // 2 pi f of the middle axis (3D)
  const uint8_t* keepx;
  const uint8_t* keepy;
  const uint8_t* keepm;       // middle axis (3D)
  float2* mid2;               // [B][n_mid2][S] fields after the middle-axis inverse transform (3D)
  int n_mid2;
  int nm;                     // points of the middle axis (3D)
  const float2* tw;           // master twiddles
  float2* dc;                 // batch-mean scratch of the KS mean removal
  float coef;                 // nonlinear coefficient
  float scale;                // 1 / (points per field)
  int C, n_aux, n_mid, n_prod;
  int integ, nstages;
  int stage;                  // stage whose nonlinear value the launch consumes; -1 primes
  int emit;                   // write the next stage's fields
  int steps;
  int B;
  int flags;
  int64_t S;
  int H;
  const uint8_t* tile_zero;  // register axis-0 pass: column tiles whose next-stage fields are zero
  int hk;                     // last-axis columns of the stage fields stored and read (FsmPlan::hk)
  int64_t wp, ms;             // row pitch and field stride of mid / prod (FsmPlan::wp, ms)
  const int32_t* tab_entry;   // per sample: its coefficient-table entry (serving), or null
  int pdl;                    // host: launch the passes as programmatic dependents (launch_pdl)
};

// The coefficient-table entry of sample b: its own entry from tab_entry when given (a serving
// engine's slots share their request's entry), else entry b of per-sample tables or the one entry.
__device__ __forceinline__ int64_t tab_batch(const StepArgs& a, int b) {
  return a.tab_entry ? (int64_t)a.tab_entry[b] : (int64_t)(a.lin_batch > 1 ? b : 0);
}

// The kernels' arguments for `batch` samples of `state` advanced by `steps` steps of plan p,
// without recording (fsm_api.cu).
StepArgs base_args(const FsmPlan* p, void* state, int32_t batch, int32_t steps);

int transform_r2c_last(int n, const float* in, float2* out, int64_t rows, const float2* tw, bool pdl, cudaStream_t st);
int transform_c2r_last(int n, const float2* in, float* out, int64_t rows, float scale, const float2* tw, bool pdl,
                       cudaStream_t st);
int transform_c2c_strided(int n, bool inverse, float2* data, int64_t outer, int64_t inner, const float2* tw, bool pdl,
                          cudaStream_t st);
// The whole real transforms of `count` fields (fsm_rfftn, fsm_irfftn), as programmatic dependents or plain launches.
int forward_real(const FsmPlan* p, int64_t count, const float* in, float2* out, bool pdl, cudaStream_t st);
int inverse_real(const FsmPlan* p, int64_t count, float2* in, float* out, bool pdl, cudaStream_t st);
int launch_nonfinite(const float2* f, int64_t count, int64_t S, int32_t* flags, cudaStream_t st);

// fsm_integrate without recording on a caller-provided workspace (fsm_api.cu).
int integrate_with_workspace(const FsmPlan* p, int32_t batch, void* state, int32_t steps, void* workspace,
                             size_t workspace_bytes, cudaStream_t st);
size_t integrate_workspace_bytes(const FsmPlan* p, int32_t batch, int32_t steps);
// fsm_integrate without recording on a caller-provided workspace; large batches may run in
// parts on the library's streams (outside stream capture), as fsm_integrate does. tab_entry
// (device, one per sample, or null): each sample's coefficient-table entry.
int integrate_on_workspace(const FsmPlan* p, int32_t batch, void* state, int32_t steps, void* workspace,
                           size_t workspace_bytes, cudaStream_t st, const int32_t* tab_entry = nullptr);
// Recompute the coefficient tables of batch entries [b0, b0 + n) for time step dt (one launch).
int set_batch_dt_range(FsmPlan* p, int32_t b0, int32_t n, double dt, cudaStream_t st);

// The three passes between the x passes in one launch where planes are small (fsm_volume_plane.cu).
bool volume_plane_applies(const FsmPlan* p);
int launch_volume_plane(const FsmPlan* p, const StepArgs& a, cudaStream_t st);
int launch_volume_axis1_inv(const FsmPlan* p, const StepArgs& a, cudaStream_t st);
int launch_volume_axis2(const FsmPlan* p, const StepArgs& a, cudaStream_t st);
int launch_volume_axis1_fwd(const FsmPlan* p, const StepArgs& a, cudaStream_t st);

int launch_line(const FsmPlan* p, const StepArgs& a, cudaStream_t st);

// The row kernel of a 2D adjoint step (fsm_adjoint_row.cu): B samples of two channels, n0 rows; half-spectrum
// arrays [..][B][2][n0][H] (th values a field pair), physical ones [..][B][2][n0][NY] (tr values).
// Forward: in[3] -> P[3] and out. Backward: in, P[3] -> out[3]. inv: 1 / points; scale: the coefficient
// (backward: times the points).
struct AdjRow {
  const float2* in;
  float* P;
  float2* out;
  const float2* tw;
  int64_t th, tr;
  float inv, scale;
  int B, n0, backward;
};
int launch_adj_row(int ny, const AdjRow& a, cudaStream_t st);

// One launch of the 1D line kernel over the samples of several plans of different lengths
// (256..4096 points, one nonlinear kind): entry j advances a[j].B samples of a[j] by a[j].steps
// steps (the same for every entry), without recording. cta0 is filled in by the launcher.
constexpr int kLineMultiMax = 8;
constexpr int kLineMultiThreads = 256;
struct LineMulti {
  StepArgs a[kLineMultiMax];
  int32_t n[kLineMultiMax];
  int32_t cta0[kLineMultiMax + 1];
  int32_t count;
};
int launch_line_multi(LineMulti& m, int kind, cudaStream_t st);

// One launch of the 2D register column (or row) pass over the samples of several plans of square
// grids (64, 128 or 256 points per axis, Convection or VorticityConvection): entry j runs the pass
// on a[j].B samples of a[j] (arguments of plane_args, stage and emit set by the caller). gx and
// cta0 are filled in by the launchers. A column launch primes every entry (stage -1) or runs a SETDRK4
// stage of every entry; others are refused.
constexpr int kPlaneMultiMax = 8;
struct PlaneMulti {
  StepArgs a[kPlaneMultiMax];
  int32_t n[kPlaneMultiMax];
  int32_t gx[kPlaneMultiMax];
  int32_t cta0[kPlaneMultiMax + 1];
  int32_t count;
};
int launch_plane_col_multi(PlaneMulti& m, int kind, cudaStream_t st);
int launch_plane_row_multi(PlaneMulti& m, int kind, cudaStream_t st);
// The plane passes' arguments for `batch` samples of `state` advanced by `steps` steps without
// recording, with the pass arrays in `workspace` laid out as fsm_integrate lays them out (fsm_api.cu).
int plane_args(const FsmPlan* p, void* state, int32_t batch, int32_t steps, void* workspace, size_t workspace_bytes,
               StepArgs* out);
// The column pass (2D; the x pass of 3D) and the row pass.
int launch_plane_col(const FsmPlan* p, const StepArgs& a, cudaStream_t st);
int launch_plane_row(const FsmPlan* p, const StepArgs& a, cudaStream_t st);
int launch_ks_mean(const FsmPlan* p, const StepArgs& a, cudaStream_t st);
int launch_pointwise(const FsmPlan* p, const StepArgs& a, cudaStream_t st);
// Parts (streams) an uncaptured integrate of `batch` samples is split into; 1: one sequence.
int split_parts(const FsmPlan* p, int batch, int steps);

// The shape of a resident 2D launch (fsm_resident.cu): cluster size, kept / other columns and rows
// per CTA, product pitch, groups per column, threads and shared memory of a CTA; steps of a launch at most.
struct ResConfig {
  int cl, ka, kb, pc, fs, rpc, threads, steps;
  bool tables;
  size_t smem;
};
// Whether a whole integrate of `batch` samples runs in the resident 2D kernel, and in which shape; `parts`:
// what the passes would run in.
bool resident_config(const FsmPlan* p, int batch, int parts, ResConfig* out);
// a.steps steps of a.B samples in one launch, frames at a.slots (device) when given.
int launch_resident(const FsmPlan* p, const ResConfig& c, const StepArgs& a, cudaStream_t st);

// Programmatic dependent launch: the grid may start (its blocks are placed, constants are loaded)
// while the one before it in the stream drains; the kernel waits in pdl_wait() before it touches
// anything that grid wrote or still reads. Every kernel launched this way calls pdl_wait() in every
// thread before its first access to global memory other than the plan's twiddles and wavenumbers,
// and pdl_trigger() late, before its last transform: triggered at the start, the next grids' waiting
// blocks took the places of running ones (512^2 x 5: 6.26 ms per 40 steps, 3D Burgers 256^3 15.2 ms
// per 4). Plain launches -> triggered late: vorticity 512^2 x 5 6.31 -> 5.33 ms, 256^2 x 64 8.61 ->
// 8.31 ms per 50 steps, 3D Burgers 64^3 x 3 5.03 -> 4.30 ms per 20, 256^3 no change.
template <class... P, class... A>
inline int launch_pdl(bool pdl, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                      const char* what, A&&... args) {
  cudaLaunchConfig_t lc = {};
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  lc.gridDim = grid;
  lc.blockDim = block;
  lc.dynamicSmemBytes = smem;
  lc.stream = st;
  lc.attrs = &at;
  lc.numAttrs = pdl ? 1 : 0;
  return cuda_check(cudaLaunchKernelEx(&lc, kernel, P(args)...), what);
}

// Raise a kernel's dynamic shared-memory limit when it needs more than 48 KB. The
// attribute is per function and per device; the size set is remembered per
// (kernel, device) so that repeated launches skip the attribute call.
SmemAttributes& smem_attributes();

template <class K>
inline int prep_smem(K kernel, size_t smem) {
  if (smem <= 48 * 1024) return FSM_OK;
  int dev = 0;
  cudaGetDevice(&dev);
  return smem_attributes().raise((const void*)kernel, dev, smem, [&] {
    return cuda_check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                      "cudaFuncSetAttribute");
  });
}

}  // namespace fsm
