// Real transforms along the contiguous last axis: two real rows travel as one complex row
// z = a + i b (forward: split with Hermitian symmetry; inverse: Z = A + i B over the Hermitian
// extension of each half spectrum). The outer axes are k_c2c_strided_r's (fsm_volume.cu).
// These serve fsm_rfftn / fsm_irfftn (FourierMesh.fft / ifft(...).real,
// mesh.py:481-491) for the initial spectrum, the returned fields and the
// recorded trajectories.
#include "fsm_internal.cuh"
#include "fsm_linefft.cuh"

namespace fsm {

// Rows of up to 512 points: a group of T lanes per pair of rows, registers from the loads to the
// stores (lanes on adjacent elements). Longer rows: T threads per pair (fsm_linefft.cuh). Bound: launch
// latency for few rows, else memory. The shared-memory Stockham passes these replaced, us per launch of
// 256^2 x 16 / 1024 x 7 / 4096 x 32: r2c 10.0 / 19.8 / 21.2, c2r 7.9 / 15.8 / 17.0; now
// 5.4 / 7.4 / 12.0 and 5.2 / 7.5 / 11.9.

// rows: [rows][N] real -> [rows][N/2+1] complex (unnormalised forward)
template <int N>
__global__ void __launch_bounds__(256) k_r2c_last(const float* __restrict__ in, float2* __restrict__ out, int64_t rows,
                                                  const float2* __restrict__ master) {
  constexpr int T = RegShape<N>::T, E = RegShape<N>::E, H = N / 2 + 1, J = N / (2 * T);
  extern __shared__ float2 smem[];
  const int lane = threadIdx.x & 31, g = threadIdx.x / T, t = threadIdx.x % T;
  load_reg_twiddles<N>(smem, master, threadIdx.x, blockDim.x);
  pdl_wait();
  in = pdl_ptr(in);
  __syncthreads();
  const int64_t r0 = ((int64_t)blockIdx.x * (blockDim.x / T) + g) * 2;
  const bool has0 = r0 < rows, has1 = r0 + 1 < rows;
  float2 v[E];
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const int n = t + T * j;
    v[j] = make_float2(has0 ? in[r0 * N + n] : 0.f, has1 ? in[(r0 + 1) * N + n] : 0.f);
  }
  pdl_trigger();
  reg_fft<N, false>(v, smem + N + g * reg_scratch<N>(), smem, t);
  const int partner_lane = (lane & ~(T - 1)) | ((T - t) & (T - 1));
#pragma unroll
  for (int j = 0; j <= J; ++j) {
    const float2 send = v[E - 1 - j];
    float2 recv;
    recv.x = __shfl_sync(0xffffffffu, send.x, partner_lane);
    recv.y = __shfl_sync(0xffffffffu, send.y, partner_lane);
    const float2 zm = cconj((t == 0) ? v[(E - j) & (E - 1)] : recv);
    const int k = t + T * j;
    if (k <= N / 2) {
      if (has0) out[r0 * H + k] = cscale(cadd(v[j], zm), 0.5f);
      if (has1) out[(r0 + 1) * H + k] = cscale(cmulmi(csub(v[j], zm)), 0.5f);
    }
  }
}

// A + i B at index k of the Hermitian extensions of two half rows.
template <int N>
__device__ __forceinline__ float2 herm_value(const float2* a, const float2* b, int k) {
  const bool hi = k > N / 2;
  const int kk = hi ? N - k : k;
  float2 A = a ? a[kk] : make_float2(0.f, 0.f), B = b ? b[kk] : make_float2(0.f, 0.f);
  if (kk == 0 || kk == N / 2) A.y = B.y = 0.f;
  if (hi) {
    A.y = -A.y;
    B.y = -B.y;
  }
  return make_float2(A.x - B.y, A.y + B.x);
}

// rows: [rows][N/2+1] complex -> [rows][N] real, times `scale`
template <int N>
__global__ void __launch_bounds__(256) k_c2r_last(const float2* __restrict__ in, float* __restrict__ out, int64_t rows,
                                                  float scale, const float2* __restrict__ master) {
  constexpr int T = RegShape<N>::T, E = RegShape<N>::E, H = N / 2 + 1;
  extern __shared__ float2 smem[];
  const int g = threadIdx.x / T, t = threadIdx.x % T;
  load_reg_twiddles<N>(smem, master, threadIdx.x, blockDim.x);
  pdl_wait();
  in = pdl_ptr(in);
  __syncthreads();
  const int64_t r0 = ((int64_t)blockIdx.x * (blockDim.x / T) + g) * 2;
  const float2* a = r0 < rows ? in + r0 * H : nullptr;
  const float2* b = r0 + 1 < rows ? in + (r0 + 1) * H : nullptr;
  float2 v[E];
#pragma unroll
  for (int j = 0; j < E; ++j) v[j] = herm_value<N>(a, b, t + T * j);
  pdl_trigger();
  reg_fft<N, true>(v, smem + N + g * reg_scratch<N>(), smem, t);
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const int n = t + T * j;
    if (a) out[r0 * N + n] = v[j].x * scale;
    if (b) out[(r0 + 1) * N + n] = v[j].y * scale;
  }
}

template <int N>
__global__ void __launch_bounds__(LineCfg<N>::T) k_r2c_line(const float* __restrict__ in, float2* __restrict__ out,
                                                            int64_t rows, const float2* __restrict__ master) {
  using Cfg = LineCfg<N>;
  constexpr int T = Cfg::T, E = Cfg::E, H = Cfg::H;
  extern __shared__ float2 smem[];
  float2 *buf0 = smem + Cfg::TW, *buf1 = buf0 + Cfg::NB;
  const int t = threadIdx.x;
  line_twiddles<N>(smem, master, t, T);
  pdl_wait();
  in = pdl_ptr(in);
  __syncthreads();
  const int64_t r0 = (int64_t)blockIdx.x * 2;
  const bool has1 = r0 + 1 < rows;
  float2 v[E];
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const int n = t + T * j;
    v[j] = make_float2(in[r0 * N + n], has1 ? in[(r0 + 1) * N + n] : 0.f);
  }
  pdl_trigger();
  line_passes<N, false, 1>(v, buf0, buf1, smem, t, 0, true);
  // Z(N - k) of the upper half through the buffer that the next exchange would take
  float2* x = (line_exchanges<N>() & 1) ? buf1 : buf0;
#pragma unroll
  for (int j = E / 2; j < E; ++j) x[line_pad(t + T * j)] = v[j];
  if (t == 0) x[0] = v[0];
  line_sync<N>(0);
#pragma unroll
  for (int j = 0; j <= E / 2; ++j) {
    const int k = t + T * j;
    if (k > N / 2) break;
    const float2 zm = cconj(x[line_pad((N - k) & (N - 1))]);
    out[r0 * H + k] = cscale(cadd(v[j], zm), 0.5f);
    if (has1) out[(r0 + 1) * H + k] = cscale(cmulmi(csub(v[j], zm)), 0.5f);
  }
}

template <int N>
__global__ void __launch_bounds__(LineCfg<N>::T) k_c2r_line(const float2* __restrict__ in, float* __restrict__ out,
                                                            int64_t rows, float scale,
                                                            const float2* __restrict__ master) {
  using Cfg = LineCfg<N>;
  constexpr int T = Cfg::T, E = Cfg::E, H = Cfg::H;
  extern __shared__ float2 smem[];
  float2 *buf0 = smem + Cfg::TW, *buf1 = buf0 + Cfg::NB;
  const int t = threadIdx.x;
  line_twiddles<N>(smem, master, t, T);
  pdl_wait();
  in = pdl_ptr(in);
  __syncthreads();
  const int64_t r0 = (int64_t)blockIdx.x * 2;
  const float2* a = in + r0 * H;
  const float2* b = r0 + 1 < rows ? a + H : nullptr;
  float2 v[E];
#pragma unroll
  for (int j = 0; j < E; ++j) v[j] = herm_value<N>(a, b, t + T * j);
  pdl_trigger();
  line_passes<N, true, 1>(v, buf0, buf1, smem, t, 0, true);
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const int n = t + T * j;
    out[r0 * N + n] = v[j].x * scale;
    if (b) out[(r0 + 1) * N + n] = v[j].y * scale;
  }
}

// Threads of a launch over `pairs` row pairs of N points: whole warps, 256 at most.
template <int N>
static int row_threads(int64_t pairs) {
  const int64_t need = pairs * RegShape<N>::T;
  return need >= 256 ? 256 : (int)((need + 31) / 32 * 32);
}

template <int N>
static int launch_r2c(const float* in, float2* out, int64_t rows, const float2* tw, bool pdl, cudaStream_t st) {
  const int64_t pairs = (rows + 1) / 2;
  if constexpr (N <= 512) {
    const int threads = row_threads<N>(pairs), groups = threads / RegShape<N>::T;
    const size_t smem = (size_t)(N + groups * reg_scratch<N>()) * sizeof(float2);
    int rc = prep_smem(k_r2c_last<N>, smem);
    if (rc) return rc;
    return launch_pdl(pdl, k_r2c_last<N>, (unsigned)((pairs + groups - 1) / groups), threads, smem, st, "k_r2c_last", in,
                      out, rows, tw);
  } else {
    const size_t smem = (size_t)(LineCfg<N>::TW + 2 * LineCfg<N>::NB) * sizeof(float2);
    int rc = prep_smem(k_r2c_line<N>, smem);
    if (rc) return rc;
    return launch_pdl(pdl, k_r2c_line<N>, (unsigned)pairs, LineCfg<N>::T, smem, st, "k_r2c_line", in, out, rows, tw);
  }
}

template <int N>
static int launch_c2r(const float2* in, float* out, int64_t rows, float scale, const float2* tw, bool pdl, cudaStream_t st) {
  const int64_t pairs = (rows + 1) / 2;
  if constexpr (N <= 512) {
    const int threads = row_threads<N>(pairs), groups = threads / RegShape<N>::T;
    const size_t smem = (size_t)(N + groups * reg_scratch<N>()) * sizeof(float2);
    int rc = prep_smem(k_c2r_last<N>, smem);
    if (rc) return rc;
    return launch_pdl(pdl, k_c2r_last<N>, (unsigned)((pairs + groups - 1) / groups), threads, smem, st, "k_c2r_last", in,
                      out, rows, scale, tw);
  } else {
    const size_t smem = (size_t)(LineCfg<N>::TW + 2 * LineCfg<N>::NB) * sizeof(float2);
    int rc = prep_smem(k_c2r_line<N>, smem);
    if (rc) return rc;
    return launch_pdl(pdl, k_c2r_line<N>, (unsigned)pairs, LineCfg<N>::T, smem, st, "k_c2r_line", in, out, rows, scale,
                      tw);
  }
}

int transform_r2c_last(int n, const float* in, float2* out, int64_t rows, const float2* tw, bool pdl, cudaStream_t st) {
  switch (n) {
    case 16: return launch_r2c<16>(in, out, rows, tw, pdl, st);
    case 32: return launch_r2c<32>(in, out, rows, tw, pdl, st);
    case 64: return launch_r2c<64>(in, out, rows, tw, pdl, st);
    case 128: return launch_r2c<128>(in, out, rows, tw, pdl, st);
    case 256: return launch_r2c<256>(in, out, rows, tw, pdl, st);
    case 512: return launch_r2c<512>(in, out, rows, tw, pdl, st);
    case 1024: return launch_r2c<1024>(in, out, rows, tw, pdl, st);
    case 2048: return launch_r2c<2048>(in, out, rows, tw, pdl, st);
    case 4096: return launch_r2c<4096>(in, out, rows, tw, pdl, st);
  }
  return set_error(FSM_ERR_UNSUPPORTED, "r2c: unsupported length " + std::to_string(n));
}

int transform_c2r_last(int n, const float2* in, float* out, int64_t rows, float scale, const float2* tw,
                       bool pdl, cudaStream_t st) {
  switch (n) {
    case 16: return launch_c2r<16>(in, out, rows, scale, tw, pdl, st);
    case 32: return launch_c2r<32>(in, out, rows, scale, tw, pdl, st);
    case 64: return launch_c2r<64>(in, out, rows, scale, tw, pdl, st);
    case 128: return launch_c2r<128>(in, out, rows, scale, tw, pdl, st);
    case 256: return launch_c2r<256>(in, out, rows, scale, tw, pdl, st);
    case 512: return launch_c2r<512>(in, out, rows, scale, tw, pdl, st);
    case 1024: return launch_c2r<1024>(in, out, rows, scale, tw, pdl, st);
    case 2048: return launch_c2r<2048>(in, out, rows, scale, tw, pdl, st);
    case 4096: return launch_c2r<4096>(in, out, rows, scale, tw, pdl, st);
  }
  return set_error(FSM_ERR_UNSUPPORTED, "c2r: unsupported length " + std::to_string(n));
}

// Per-field NaN/Inf flags: one block per field.
__global__ void k_nonfinite(const float2* __restrict__ f, int64_t S, int32_t* __restrict__ flags) {
  const float2* p = f + (int64_t)blockIdx.x * S;
  int bad = 0;
  for (int64_t i = threadIdx.x; i < S; i += blockDim.x) {
    const float2 v = p[i];
    bad |= !(isfinite(v.x) && isfinite(v.y));
  }
  bad = __syncthreads_or(bad);
  if (threadIdx.x == 0) flags[blockIdx.x] = bad ? 1 : 0;
}

int launch_nonfinite(const float2* f, int64_t count, int64_t S, int32_t* flags, cudaStream_t st) {
  if (count <= 0) return FSM_OK;
  k_nonfinite<<<(unsigned)count, 256, 0, st>>>(f, S, flags);
  return cuda_check(cudaGetLastError(), "k_nonfinite");
}

}  // namespace fsm
