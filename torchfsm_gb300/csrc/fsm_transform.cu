// Real transforms along the contiguous last axis: two real rows travel as one complex row
// z = a + i b (forward: split with Hermitian symmetry; inverse: Z = A + i B over the Hermitian
// extension of each half spectrum). The outer axes are k_c2c_strided_r's (fsm_volume.cu).
// These serve fsm_rfftn / fsm_irfftn (FourierMesh.fft / ifft(...).real,
// mesh.py:481-491) for the initial spectrum, the returned fields and the
// recorded trajectories.
#include "fsm_internal.cuh"

namespace fsm {

template <int N>
struct RowCfg {
  static constexpr int G = (N / 16 < 32) ? 32 : N / 16;
  static constexpr bool BLOCK = G > 32;
  static constexpr int GROUPS = BLOCK ? 1 : 8;
  static constexpr int THREADS = G * GROUPS;
  static constexpr size_t SMEM = (size_t)(GROUPS + 1) * N * sizeof(float2);
};

// rows: [rows][N] real -> [rows][N/2+1] complex (unnormalised forward)
template <int N>
__global__ void __launch_bounds__(RowCfg<N>::THREADS) k_r2c_last(const float* __restrict__ in, float2* __restrict__ out,
                                                                  int64_t rows, const float2* __restrict__ master) {
  using Cfg = RowCfg<N>;
  constexpr int H = N / 2 + 1;
  extern __shared__ float2 smem[];
  float2* tw = smem;
  const int g = threadIdx.x / Cfg::G;
  const int t = threadIdx.x % Cfg::G;
  float2* z = smem + N + g * N;
  load_twiddles(tw, master, kTwiddleMax, N, threadIdx.x, Cfg::THREADS);
  pdl_wait();
  in = pdl_ptr(in);
  const int64_t r0 = ((int64_t)blockIdx.x * Cfg::GROUPS + g) * 2;
  const bool has0 = r0 < rows, has1 = r0 + 1 < rows;
  for (int n = t; n < N; n += Cfg::G) {
    const float a = has0 ? in[r0 * N + n] : 0.f;
    const float b = has1 ? in[(r0 + 1) * N + n] : 0.f;
    z[n] = make_float2(a, b);
  }
  __syncthreads();
  pdl_trigger();
  fft<N, Cfg::G, Cfg::BLOCK, false>(z, tw, t);
  for (int k = t; k < H; k += Cfg::G) {
    const float2 zk = z[k];
    const float2 zm = cconj(z[(N - k) & (N - 1)]);
    if (has0) out[r0 * H + k] = cscale(cadd(zk, zm), 0.5f);
    if (has1) out[(r0 + 1) * H + k] = cscale(cmulmi(csub(zk, zm)), 0.5f);
  }
}

// rows: [rows][N/2+1] complex -> [rows][N] real, times `scale`
template <int N>
__global__ void __launch_bounds__(RowCfg<N>::THREADS) k_c2r_last(const float2* __restrict__ in, float* __restrict__ out,
                                                                  int64_t rows, float scale,
                                                                  const float2* __restrict__ master) {
  using Cfg = RowCfg<N>;
  constexpr int H = N / 2 + 1;
  extern __shared__ float2 smem[];
  float2* tw = smem;
  const int g = threadIdx.x / Cfg::G;
  const int t = threadIdx.x % Cfg::G;
  float2* z = smem + N + g * N;
  load_twiddles(tw, master, kTwiddleMax, N, threadIdx.x, Cfg::THREADS);
  pdl_wait();
  in = pdl_ptr(in);
  const int64_t r0 = ((int64_t)blockIdx.x * Cfg::GROUPS + g) * 2;
  const bool has0 = r0 < rows, has1 = r0 + 1 < rows;
  for (int k = t; k < H; k += Cfg::G) {
    float2 A = has0 ? in[r0 * H + k] : make_float2(0.f, 0.f);
    float2 B = has1 ? in[(r0 + 1) * H + k] : make_float2(0.f, 0.f);
    if (k == 0 || k == N / 2) {
      A.y = 0.f;
      B.y = 0.f;
    }
    z[k] = make_float2(A.x - B.y, A.y + B.x);  // A + i B
    if (k > 0 && k < N / 2) z[N - k] = make_float2(A.x + B.y, B.x - A.y);  // conj(A) + i conj(B)
  }
  __syncthreads();
  pdl_trigger();
  fft<N, Cfg::G, Cfg::BLOCK, true>(z, tw, t);
  for (int n = t; n < N; n += Cfg::G) {
    const float2 v = z[n];
    if (has0) out[r0 * N + n] = v.x * scale;
    if (has1) out[(r0 + 1) * N + n] = v.y * scale;
  }
}

template <int N>
static int launch_r2c(const float* in, float2* out, int64_t rows, const float2* tw, bool pdl, cudaStream_t st) {
  using Cfg = RowCfg<N>;
  int rc = prep_smem(k_r2c_last<N>, Cfg::SMEM);
  if (rc) return rc;
  const int64_t pairs = (rows + 1) / 2;
  const int64_t blocks = (pairs + Cfg::GROUPS - 1) / Cfg::GROUPS;
  return launch_pdl(pdl, k_r2c_last<N>, (unsigned)blocks, Cfg::THREADS, Cfg::SMEM, st, "k_r2c_last", in, out, rows, tw);
}

template <int N>
static int launch_c2r(const float2* in, float* out, int64_t rows, float scale, const float2* tw, bool pdl, cudaStream_t st) {
  using Cfg = RowCfg<N>;
  int rc = prep_smem(k_c2r_last<N>, Cfg::SMEM);
  if (rc) return rc;
  const int64_t pairs = (rows + 1) / 2;
  const int64_t blocks = (pairs + Cfg::GROUPS - 1) / Cfg::GROUPS;
  return launch_pdl(pdl, k_c2r_last<N>, (unsigned)blocks, Cfg::THREADS, Cfg::SMEM, st, "k_c2r_last", in, out, rows,
                    scale, tw);
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
