// The y and z passes of a 3D velocity stage in one kernel, a CTA per (sample, x) plane: the plane's
// stage fields and products stay in shared memory between the y inverse transforms, the z pass and
// the y forward transforms, which are three launches and 24 field passes through memory otherwise
// (fsm_volume.cu: k_axis1_inv_r, k_axis2_r, k_c2c_strided_r). Planes of up to 4096 points.
// Bound: the latency of the transforms' chains at 16 warps per SM. Three launches -> one, us per step of
// 3D Burgers: 32^3 x 1 113 -> 46, x 64 874 -> 450; 64^3 x 1 140 -> 80, x 3 217 -> 149, x 12 692 -> 445;
// 64 x 128 x 32 x 2 271 -> 118. Always taken where it fits.
#include "fsm_internal.cuh"
#include "fsm_regfft.cuh"

namespace fsm {

constexpr int kPlaneThreads = 512;

template <int NY, int NZ>
struct VolPlaneCfg {
  static constexpr int TY = RegShape<NY>::T, EY = RegShape<NY>::E, TZ = RegShape<NZ>::T, EZ = RegShape<NZ>::E;
  static constexpr int H = NZ / 2 + 1, HK = NZ / 3 + 1;
  static constexpr int RP = NY + 1;  // column pitch
  static constexpr int MID = 9 * HK * RP, PROD = 3 * H * RP;
  static constexpr int SY = (kPlaneThreads / TY) * reg_scratch<NY>(), SZ = (kPlaneThreads / TZ) * reg_scratch<NZ>();
  static constexpr int SCR = SY > SZ ? SY : SZ;
  static constexpr size_t SMEM = (size_t)(NY + NZ + MID + PROD + SCR) * sizeof(float2);
};

// Z = A + i B over the Hermitian extension of a row of two fields (columns RP apart; a null field is
// zero), `da` / `db` applying i kz.
template <int NZ, int RP>
__device__ __forceinline__ void plane_row(float2 (&Z)[RegShape<NZ>::E], const float2* fa, const float2* fb, bool da,
                                          bool db, const float* __restrict__ kz, int t) {
  constexpr int T = RegShape<NZ>::T, E = RegShape<NZ>::E, HK = NZ / 3 + 1;
#pragma unroll
  for (int j = 0; j < E; ++j) {
    Z[j] = make_float2(0.f, 0.f);
    if (reg_dead<NZ, T, HK>(j)) continue;
    const int k = t + T * j;
    const bool hi = k > NZ / 2;
    const int kk = hi ? NZ - k : k;
    if (kk < HK) {
      float2 A = fa[kk * RP], B = fb[kk * RP];
      if (da) A = cscale(cmuli(A), kz[kk]);
      if (db) B = cscale(cmuli(B), kz[kk]);
      if (kk == 0) {
        A.y = 0.f;
        B.y = 0.f;
      }
      if (hi) {
        A.y = -A.y;
        B.y = -B.y;
      }
      Z[j] = make_float2(A.x - B.y, A.y + B.x);
    }
  }
}

// Split the transform of p0 + i p1 (lane t holds K = t + T j) into half spectra at columns RP apart.
template <int NZ, int RP>
__device__ __forceinline__ void plane_split(const float2 (&zp)[RegShape<NZ>::E], int t, int lane, bool on, float2* out0,
                                            float2* out1) {
  constexpr int T = RegShape<NZ>::T, E = RegShape<NZ>::E, J = NZ / (2 * T);
  const int partner_lane = (lane & ~(T - 1)) | ((T - t) & (T - 1));
#pragma unroll
  for (int j = 0; j <= J; ++j) {
    const float2 send = zp[E - 1 - j];
    float2 recv;
    recv.x = __shfl_sync(0xffffffffu, send.x, partner_lane);
    recv.y = __shfl_sync(0xffffffffu, send.y, partner_lane);
    const float2 zm = cconj((t == 0) ? zp[(E - j) & (E - 1)] : recv);
    const int k = t + T * j;
    if (k <= NZ / 2 && on) {
      out0[k * RP] = cscale(cadd(zp[j], zm), 0.5f);
      if (out1) out1[k * RP] = cscale(cmulmi(csub(zp[j], zm)), 0.5f);
    }
  }
}

template <int NY, int NZ>
__global__ void __launch_bounds__(kPlaneThreads) k_volume_plane(StepArgs a) {
  using Cfg = VolPlaneCfg<NY, NZ>;
  constexpr int H = Cfg::H, HK = Cfg::HK, RP = Cfg::RP;
  extern __shared__ float2 smem[];
  float2* twy = smem;
  float2* twz = twy + NY;
  float2* mid = twz + NZ;       // [9][HK][RP]: per channel c, 3c: u_c, 3c + 1: d_x u_c, 3c + 2: d_y u_c
  float2* prod = mid + Cfg::MID;  // [3][H][RP]
  float2* scr = prod + Cfg::PROD;
  const int lane = threadIdx.x & 31;
  const int x = blockIdx.x, b = blockIdx.y;
  const int64_t S = a.S, plane = (int64_t)NY * H;
  load_reg_twiddles<NY>(twy, a.tw, threadIdx.x, kPlaneThreads);
  load_reg_twiddles<NZ>(twz, a.tw, threadIdx.x, kPlaneThreads);
  pdl_wait();
  __syncthreads();
  {
    // y inverse: a group per (channel, kept column); columns fastest, so that a warp's groups read
    // adjacent words of a row
    constexpr int T = Cfg::TY, E = Cfg::EY, GPW = 32 / T, ITEMS = 3 * HK;
    const int t = lane % T, sub = lane / T;
    float2* sc = scr + (threadIdx.x / T) * reg_scratch<NY>();
#pragma unroll 1
    for (int base = (threadIdx.x >> 5) * GPW; base < ITEMS; base += kPlaneThreads / T) {
      const int item = base + sub < ITEMS ? base + sub : ITEMS - 1;  // spare groups repeat the last one
      const int c = item / HK, col = item % HK;
      const float2* in0 = a.mid + ((int64_t)b * a.n_mid + 2 * c) * S + x * plane + col;
      const float2* in1 = in0 + S;
      float2* out = mid + (3 * c * HK + col) * RP;
      float2 v[E], w[E], d[E];
#pragma unroll
      for (int j = 0; j < E; ++j) {
        const int row = t + T * j;
        const bool keep = a.keepm[row];  // the x pass stores the kept rows alone
        v[j] = keep ? in0[(int64_t)row * H] : make_float2(0.f, 0.f);
        d[j] = keep ? in1[(int64_t)row * H] : make_float2(0.f, 0.f);
        w[j] = cscale(cmuli(v[j]), a.km[row]);
      }
      reg_fft<NY, true>(v, sc, twy, t);
      reg_fft<NY, true>(d, sc, twy, t);
      reg_fft<NY, true>(w, sc, twy, t);
#pragma unroll
      for (int j = 0; j < E; ++j) {
        out[t + T * j] = v[j];
        out[HK * RP + t + T * j] = d[j];
        out[2 * HK * RP + t + T * j] = w[j];
      }
    }
  }
  __syncthreads();
  {
    // z: a group per row, the products of k_axis2_r in its order
    constexpr int T = Cfg::TZ, E = Cfg::EZ, GPW = 32 / T, F = HK * RP;
    const int t = lane % T, sub = lane / T;
    const float* kz = a.ky;
    float2* sc = scr + (threadIdx.x / T) * reg_scratch<NZ>();
#pragma unroll 1
    for (int base = (threadIdx.x >> 5) * GPW; base < NY; base += kPlaneThreads / T) {
      const bool on = base + sub < NY;
      const int row = on ? base + sub : NY - 1;
      const float2* m = mid + row;
      float2 Z[E];
      float u0[E], u1[E], u2[E], c0[E], c1[E], c2[E];
      plane_row<NZ, RP>(Z, m, m + 3 * F, false, false, kz, t);  // u0 + i u1
      reg_fft<NZ, true>(Z, sc, twz, t);
#pragma unroll
      for (int j = 0; j < E; ++j) {
        u0[j] = Z[j].x;
        u1[j] = Z[j].y;
      }
      plane_row<NZ, RP>(Z, m + 6 * F, m + F, false, false, kz, t);  // u2 + i dx u0
      reg_fft<NZ, true>(Z, sc, twz, t);
#pragma unroll
      for (int j = 0; j < E; ++j) {
        u2[j] = Z[j].x;
        c0[j] = u0[j] * Z[j].y;
      }
      plane_row<NZ, RP>(Z, m + 2 * F, m, false, true, kz, t);  // dy u0 + i dz u0
      reg_fft<NZ, true>(Z, sc, twz, t);
#pragma unroll
      for (int j = 0; j < E; ++j) c0[j] += u1[j] * Z[j].x + u2[j] * Z[j].y;
      plane_row<NZ, RP>(Z, m + 4 * F, m + 5 * F, false, false, kz, t);  // dx u1 + i dy u1
      reg_fft<NZ, true>(Z, sc, twz, t);
#pragma unroll
      for (int j = 0; j < E; ++j) c1[j] = u0[j] * Z[j].x + u1[j] * Z[j].y;
      plane_row<NZ, RP>(Z, m + 3 * F, m + 7 * F, true, false, kz, t);  // dz u1 + i dx u2
      reg_fft<NZ, true>(Z, sc, twz, t);
#pragma unroll
      for (int j = 0; j < E; ++j) {
        c1[j] += u2[j] * Z[j].x;
        c2[j] = u0[j] * Z[j].y;
      }
      plane_row<NZ, RP>(Z, m + 8 * F, m + 6 * F, false, true, kz, t);  // dy u2 + i dz u2
      reg_fft<NZ, true>(Z, sc, twz, t);
#pragma unroll
      for (int j = 0; j < E; ++j) {
        c2[j] += u1[j] * Z[j].x + u2[j] * Z[j].y;
        Z[j] = make_float2(c0[j], c1[j]);
      }
      reg_fft<NZ, false>(Z, sc, twz, t);
      plane_split<NZ, RP>(Z, t, lane, on, prod + row, prod + H * RP + row);
#pragma unroll
      for (int j = 0; j < E; ++j) Z[j] = make_float2(c2[j], 0.f);
      reg_fft<NZ, false>(Z, sc, twz, t);
      plane_split<NZ, RP>(Z, t, lane, on, prod + 2 * H * RP + row, nullptr);
    }
  }
  __syncthreads();
  pdl_trigger();
  {
    // y forward: a group per (channel, column)
    constexpr int T = Cfg::TY, E = Cfg::EY, GPW = 32 / T, ITEMS = 3 * H;
    const int t = lane % T, sub = lane / T;
    float2* sc = scr + (threadIdx.x / T) * reg_scratch<NY>();
#pragma unroll 1
    for (int base = (threadIdx.x >> 5) * GPW; base < ITEMS; base += kPlaneThreads / T) {
      const bool on = base + sub < ITEMS;
      const int item = on ? base + sub : ITEMS - 1;
      const int c = item / H, col = item % H;
      const float2* in = prod + item * RP;
      float2 v[E];
#pragma unroll
      for (int j = 0; j < E; ++j) v[j] = in[t + T * j];
      reg_fft<NY, false>(v, sc, twy, t);
      float2* out = a.prod + ((int64_t)b * a.n_prod + c) * S + x * plane + col;
      if (on) {
#pragma unroll
        for (int j = 0; j < E; ++j) out[(int64_t)(t + T * j) * H] = v[j];
      }
    }
  }
}

namespace {
template <int NY, int NZ>
int launch_plane(int n0, const StepArgs& a, cudaStream_t st) {
  constexpr size_t smem = VolPlaneCfg<NY, NZ>::SMEM;
  int rc = prep_smem(k_volume_plane<NY, NZ>, smem);
  if (rc) return rc;
  return launch_pdl(a.pdl, k_volume_plane<NY, NZ>, dim3((unsigned)n0, (unsigned)a.B), kPlaneThreads, smem, st,
                    "k_volume_plane", a);
}

template <int NY>
int plane_row_dispatch(int nz, int n0, const StepArgs& a, cudaStream_t st) {
  switch (nz) {
    case 16: return launch_plane<NY, 16>(n0, a, st);
    case 32:
      if constexpr (NY <= 128) return launch_plane<NY, 32>(n0, a, st);
      break;
    case 64:
      if constexpr (NY <= 64) return launch_plane<NY, 64>(n0, a, st);
      break;
    case 128:
      if constexpr (NY <= 32) return launch_plane<NY, 128>(n0, a, st);
      break;
    case 256:
      if constexpr (NY <= 16) return launch_plane<NY, 256>(n0, a, st);
      break;
  }
  return set_error(FSM_ERR_UNSUPPORTED, "3D plane kernel: unsupported size");
}
}  // namespace

// The velocity programs (Convection, the Leray projection) with the 2/3 rule's kept columns, planes of up
// to 4096 points (what fits one SM's shared memory; 256 x 16 does not).
bool volume_plane_applies(const FsmPlan* p) {
  return (p->nl == FSM_NL_CONVECTION || p->nl == FSM_NL_LERAY) && p->hk == p->n[2] / 3 + 1 &&
         p->n[1] <= 128 && (int64_t)p->n[1] * p->n[2] <= 4096;
}

int launch_volume_plane(const FsmPlan* p, const StepArgs& a, cudaStream_t st) {
  switch (p->n[1]) {
    case 16: return plane_row_dispatch<16>(p->n[2], p->n[0], a, st);
    case 32: return plane_row_dispatch<32>(p->n[2], p->n[0], a, st);
    case 64: return plane_row_dispatch<64>(p->n[2], p->n[0], a, st);
    case 128: return plane_row_dispatch<128>(p->n[2], p->n[0], a, st);
  }
  return set_error(FSM_ERR_UNSUPPORTED, "3D plane kernel: unsupported size");
}

}  // namespace fsm
