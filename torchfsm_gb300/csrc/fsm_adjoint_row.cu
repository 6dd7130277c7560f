// The last-axis work of a 2D adjoint step (fsm_adjoint.cu) in one kernel per stage and direction: the
// inverse transforms of a row's fields, the products and the forward transforms of the results, a
// group of T lanes per row with the row in registers. As separate transforms and elementwise kernels
// these were three launches each way and wrote the products to memory and read them back.
// Bound: launch latency and the chain of four transforms (128^2 x 16: the step's arrays stay in L2).
// Kernel launches of a step 49 -> 33; one fit iteration of 50 steps at 128^2 x 16: 22.4 -> 20.5 ms.
#include "fsm_internal.cuh"
#include "fsm_plane_reg.cuh"

namespace fsm {

// Z = A + i B of one half row of two fields, over its Hermitian extension.
template <int NY>
__device__ __forceinline__ void adj_row_load(float2 (&Z)[RegShape<NY>::E], const float2* fa, const float2* fb, int t) {
  constexpr int T = RegShape<NY>::T, E = RegShape<NY>::E;
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const int k = t + T * j;
    const bool hi = k > NY / 2;
    const int kk = hi ? NY - k : k;
    Z[j] = herm_z(fa[kk], fb[kk], kk == 0 || kk == NY / 2, hi);
  }
}

template <int NY>
__global__ void __launch_bounds__(256) k_adj_row(AdjRow a) {
  constexpr int T = RegShape<NY>::T, E = RegShape<NY>::E, H = NY / 2 + 1;
  extern __shared__ float2 smem[];
  const int lane = threadIdx.x & 31, g = threadIdx.x / T, t = threadIdx.x % T, groups = blockDim.x / T;
  float2* twt = smem;
  float2* scr = smem + NY + g * reg_scratch<NY>();
  load_reg_twiddles<NY>(twt, a.tw, threadIdx.x, blockDim.x);
  pdl_wait();
  __syncthreads();
  // a power of two of rows: the groups of a launch cover them without a remainder
  const int64_t row = (int64_t)blockIdx.x * groups + g;
  const int64_t b = row / a.n0, x = row % a.n0;
  const int64_t h0 = ((b * 2) * a.n0 + x) * H, h1 = h0 + (int64_t)a.n0 * H;    // half rows of the channels
  const int64_t p0 = ((b * 2) * a.n0 + x) * NY, p1 = p0 + (int64_t)a.n0 * NY;  // their physical rows
  float2 Z[E];
  if (!a.backward) {
    // u, d_x u, d_y u of both channels -> P; coef sum_i u_i d_i u_c -> out
    float2 u[E], acc[E];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      adj_row_load<NY>(Z, a.in + i * a.th + h0, a.in + i * a.th + h1, t);
      reg_fft<NY, true>(Z, scr, twt, t);
      float* P = a.P + i * a.tr;
#pragma unroll
      for (int j = 0; j < E; ++j) {
        const float2 v = cscale(Z[j], a.inv);
        P[p0 + t + T * j] = v.x;
        P[p1 + t + T * j] = v.y;
        if (i == 0) u[j] = v;
        else if (i == 1) acc[j] = cscale(v, u[j].x);
        else acc[j] = cscale(make_float2(fmaf(u[j].y, v.x, acc[j].x), fmaf(u[j].y, v.y, acc[j].y)), a.scale);
      }
    }
    pdl_trigger();
    reg_fft<NY, false>(acc, scr, twt, t);
    split_store_r<NY>(acc, t, lane, a.out + h0, a.out + h1);
  } else {
    // w_c = scale irfft(in_c); sum_c' w_c' d_c u_c' and u_i w_c -> out (three pairs of fields)
    adj_row_load<NY>(Z, a.in + h0, a.in + h1, t);
    reg_fft<NY, true>(Z, scr, twt, t);
    float2 w[E];
#pragma unroll
    for (int j = 0; j < E; ++j) w[j] = cscale(cscale(Z[j], a.inv), a.scale);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
      for (int j = 0; j < E; ++j) {
        const int64_t q0 = p0 + t + T * j, q1 = p1 + t + T * j;
        if (i == 0) {
          const float* gx = a.P + a.tr;
          const float* gy = a.P + 2 * a.tr;
          Z[j] = make_float2(fmaf(w[j].y, gx[q1], w[j].x * gx[q0]), fmaf(w[j].y, gy[q1], w[j].x * gy[q0]));
        } else {
          Z[j] = cscale(w[j], a.P[i == 1 ? q0 : q1]);
        }
      }
      if (i == 2) pdl_trigger();
      reg_fft<NY, false>(Z, scr, twt, t);
      split_store_r<NY>(Z, t, lane, a.out + i * a.th + h0, a.out + i * a.th + h1);
    }
  }
}

namespace {
template <int NY>
int launch_row(const AdjRow& a, cudaStream_t st) {
  int groups = 256 / RegShape<NY>::T;
  const int64_t rows = (int64_t)a.B * a.n0;  // n0 >= 16
  while (rows % groups) groups /= 2;
  const size_t smem = (size_t)(NY + groups * reg_scratch<NY>()) * sizeof(float2);
  int rc = prep_smem(k_adj_row<NY>, smem);
  if (rc) return rc;
  return launch_pdl(true, k_adj_row<NY>, (unsigned)(rows / groups), groups * RegShape<NY>::T, smem, st, "k_adj_row", a);
}
}  // namespace

int launch_adj_row(int ny, const AdjRow& a, cudaStream_t st) {
  switch (ny) {
    case 16: return launch_row<16>(a, st);
    case 32: return launch_row<32>(a, st);
    case 64: return launch_row<64>(a, st);
    case 128: return launch_row<128>(a, st);
    case 256: return launch_row<256>(a, st);
    case 512: return launch_row<512>(a, st);
  }
  return set_error(FSM_ERR_UNSUPPORTED, "adjoint row: unsupported length");
}

}  // namespace fsm
