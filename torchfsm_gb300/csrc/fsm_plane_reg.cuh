// Device bodies of the register-FFT 2D column and row passes (16..512 points per axis; the column
// pass is also the 3D x pass), shared by the kernels of one plan (fsm_plane_col.cu,
// fsm_plane_row.cu), the kernels that advance several plans in one launch (fsm_plane_multi.cu) and,
// in parts, the resident 2D kernel (fsm_resident.cuh).
//
// Each stage of an exponential Runge-Kutta (or Runge-Kutta) scheme on half spectra [B][C][NX][H],
// H = NY/2 + 1, is two passes over the batch:
//  column pass (x): forward transform of the products left by the row pass -> N_s (plus the Leray
//    projection, plus the source); the stage update, recording when a step completes; the next
//    stage's fields (2/3 mask, 1/(NX NY), x derivatives, streamfunction) and their inverse transform.
//  row pass (y): c2r of those fields (y derivatives), the product, r2c.
// Programs (nonlinear term, operator/_base.py:375-403; input masked only):
//  FSM_NL_VORTICITY  psi = -w/lap (1 at k = 0), u = (d_y psi, -d_x psi),
//                    product u.grad(w) (operator/dedicated/_navier_stokes.py:40-46)
//                    mid: psi, i kx psi, w, i kx w
//  FSM_NL_CONVECTION (u.grad)u with C = 2 (operator/generic/_convection.py:43-46)
//                    mid: u0, i kx u0, u1, i kx u1; products conv0 + i conv1
//  FSM_NL_LERAY      convection, then N = i k p - conv, p = (i k . conv)/lap
//                    (operator/dedicated/_navier_stokes.py:246-254)
//  FSM_NL_KS         0.5|grad phi|^2, mean over the batch removed on request
//                    (operator/dedicated/_ks_convection.py:27-38); mid: phi, i kx phi
// The transforms run in registers (fsm_regfft.cuh), so each 1D transform touches shared memory once
// (512 points: twice).
//
// Row pass: a group of T lanes owns a pair of rows. It loads the mid fields
// straight from global memory into the transform layout (the Hermitian
// extension k > NY/2 comes from the mirrored entry), runs the inverse
// transforms, forms the physical product in registers, runs the forward
// transform of the two rows' products packed as one complex row and splits
// the half spectra with one shuffle per output register.
//
// Column pass: a CTA owns W = 256/T adjacent ky columns of one sample; a thread holds T-strided rows
// of one column in registers from the products through the update to the next-stage fields, with a
// warp's lanes on adjacent columns, so every global access is coalesced without staging.
#pragma once

#include "fsm_colfft.cuh"
#include "fsm_internal.cuh"
#include "fsm_regfft.cuh"

namespace fsm {

template <int KIND, int DIM>
struct RegKind {
  // channels of the state
  static constexpr int C = (KIND == FSM_NL_CONVECTION || KIND == FSM_NL_LERAY) ? DIM : 1;
  // channels whose stage update runs together (the Leray projection mixes all of them)
  static constexpr int CG = (KIND == FSM_NL_LERAY) ? C : 1;
  // mid fields written per channel group
  static constexpr int NMG = (KIND == FSM_NL_VORTICITY) ? 4 : 2 * CG;
};

// Wavenumbers and dealias factor of the point (row, inner index j). 2D: j is
// the last-axis index; 3D: j = jm * H + jl (middle, last axis).
template <int DIM>
struct PointK {
  float kx, ky, kz;  // ky: second axis, kz: third axis (3D)
  float mask;
};

template <int DIM>
__device__ __forceinline__ PointK<DIM> point_k(const StepArgs& a, int row, int64_t j) {
  PointK<DIM> p;
  p.kx = a.kx[row];
  if (DIM == 2) {
    p.ky = a.ky[j];
    p.kz = 0.f;
    p.mask = (float)(a.keepx[row] & a.keepy[j]);
  } else {
    const int jm = (int)(j / a.H), jl = (int)(j % a.H);
    p.ky = a.km[jm];
    p.kz = a.ky[jl];
    p.mask = (float)(a.keepx[row] & a.keepm[jm] & a.keepy[jl]);
  }
  p.mask *= a.scale;
  return p;
}

// Leray projection of the convection term at one point: N_c = i k_c p - conv_c,
// p = (sum_i i k_i conv_i) / lap (1 where lap == 0), operator/dedicated/_navier_stokes.py:246-254.
// The state stores only the last axis' first half, so at points whose mirror -k
// is not stored (last-axis index strictly inside) the kernel must advance the
// Hermitian part (N(k) + conj N(-k)) / 2, which is what ifftn(...).real of the
// reference's state follows. Where a non-last axis sits at its Nyquist index its
// wavenumber does not change sign under k -> -k, and that Hermitian part is the
// projection restricted to axes with the same Nyquist status as c.
// 1 / lap, 1 where lap == 0.
__device__ __forceinline__ float inv_laplacian(float kx, float ky, float kz, int dim) {
  float lap = 0.f;
  lap -= kx * kx;
  lap -= ky * ky;
  if (dim == 3) lap -= kz * kz;
  return (lap == 0.f) ? 1.f : 1.f / lap;
}

template <int DIM, int CG>
__device__ __forceinline__ void nv_leray_il(float2 (&nv)[CG], const PointK<DIM>& pk, int row, int64_t j,
                                            const StepArgs& a, int nx, float il) {
  const float kk[3] = {pk.kx, pk.ky, pk.kz};
  float sgn[3] = {1.f, 1.f, 1.f};
  int jl, jm = 0;
  if (DIM == 2) {
    jl = (int)j;
  } else {
    jm = (int)(j / a.H);
    jl = (int)(j % a.H);
  }
  const bool inside = jl > 0 && jl < a.H - 1;
  if (inside) {
    if (row == nx / 2) sgn[0] = -1.f;
    if (DIM == 3 && jm == a.nm / 2) sgn[1] = -1.f;
  }
  float2 out[CG];
#pragma unroll
  for (int c = 0; c < CG; ++c) {
    float2 div = make_float2(0.f, 0.f);
#pragma unroll
    for (int f = 0; f < CG; ++f)
      if (sgn[f] == sgn[c]) div = cadd(div, cscale(cmuli(nv[f]), kk[f]));
    out[c] = csub(cscale(cmuli(cscale(div, il)), kk[c]), nv[c]);
  }
#pragma unroll
  for (int c = 0; c < CG; ++c) nv[c] = out[c];
}

template <int DIM, int CG>
__device__ __forceinline__ void nv_leray(float2 (&nv)[CG], const PointK<DIM>& pk, int row, int64_t j,
                                         const StepArgs& a, int nx) {
  nv_leray_il<DIM, CG>(nv, pk, row, j, a, nx, inv_laplacian(pk.kx, pk.ky, pk.kz, DIM));
}

// One SETDRK4 stage at one point from its operands already in registers (the recurrences of
// etd_stage_c): ua is u at stages 0 and 1, acc at stages 2 and 3; ub is acc at stage 1, q at stage
// 2. The running sums the stage writes are returned in acc / q, the new state (stage 3) in the
// return value, which is otherwise the next stage's input.
template <int S>
__device__ __forceinline__ float2 setdrk4_pre(float2 nv, float2 ua, float2 ub, const float2* __restrict__ tab,
                                              int64_t ts, float2& acc, float2& q) {
  if (S == 0) {
    const float2 Em1 = tab[0], E2m1 = tab[ts], c1 = tab[2 * ts], c4 = tab[3 * ts];
    const float2 a1 = cfma(c1, nv, cexpmul(E2m1, ua));
    acc = cfma(c4, nv, cexpmul(Em1, ua));
    q = cfma(make_float2(-c1.x, -c1.y), nv, cexpmul(E2m1, a1));
    return a1;
  } else if (S == 1) {
    const float2 E2m1 = tab[ts], c1 = tab[2 * ts], c5 = tab[4 * ts];
    acc = cfma(cscale(c5, 2.f), nv, ub);
    return cfma(c1, nv, cexpmul(E2m1, ua));
  } else if (S == 2) {
    const float2 c1 = tab[2 * ts], c5 = tab[4 * ts];
    acc = cfma(cscale(c5, 2.f), nv, ua);
    return cfma(cscale(c1, 2.f), nv, ub);
  } else {
    return cfma(tab[5 * ts], nv, ua);
  }
}

// The SETDRK4 stage update of a thread's points (rows t + T j of its column) of a one-channel group,
// N_s in v, the next stage's input out. o1 holds the operand loaded ahead of the forward transform
// (u at stages 0 and 1, acc at stages 2 and 3), so that its latency passes behind the transform.
template <int NX, int KIND, int DIM, int STG>
__device__ __forceinline__ void axis0_update_hoisted(const StepArgs& a, float2 (&v)[RegShape<NX>::E],
                                                     const float2 (&o1)[RegShape<NX>::E], int b, int64_t j0, int t,
                                                     int cg, bool last) {
  using K = RegKind<KIND, DIM>;
  constexpr int T = RegShape<NX>::T, E = RegShape<NX>::E, C = K::C;
  const int64_t S = a.S, inner = S / NX;
  const int64_t off = ((int64_t)b * C + cg) * S + j0;
  float2* __restrict__ up = a.state + off;
  float2* __restrict__ accp = a.aux + ((int64_t)b * a.n_aux * C + cg) * S + j0;
  float2* __restrict__ qp = accp + (int64_t)C * S;
  const float2* __restrict__ tab = a.tab + (tab_batch(a, b) * a.lin_ch + (a.lin_ch > 1 ? cg : 0)) * S + j0;
  const float2* __restrict__ srcp = a.src ? a.src + ((int64_t)(a.src_batch > 1 ? b : 0) * C + cg) * S + j0 : nullptr;
  const float2* __restrict__ o2p = (STG == 1) ? accp : qp;
  // The operands of HALF points are loaded in one batch (one round of memory latency each half). The
  // SETDRK coefficients are real (k_phi_tables): only the exponentials are read as complex.
  constexpr int HALF = E > 8 ? (DIM == 2 && STG <= 1 ? 4 : 8) : E;
#pragma unroll
  for (int h0 = 0; h0 < E; h0 += HALF) {
    float2 o2[HALF], em[HALF], e2[HALF];
    float ca[HALF], cb[HALF];
#pragma unroll
    for (int i = 0; i < HALF; ++i) {
      const int64_t r = (int64_t)(t + T * (h0 + i)) * inner;
      if (STG == 1 || STG == 2) o2[i] = o2p[r];
      if (STG == 0) em[i] = tab[r];
      if (STG <= 1) e2[i] = tab[r + a.ts];
      if (STG <= 2) ca[i] = tab[r + 2 * a.ts].x;
      if (STG == 0) cb[i] = tab[r + 3 * a.ts].x;
      if (STG == 1 || STG == 2) cb[i] = tab[r + 4 * a.ts].x;
      if (STG == 3) cb[i] = tab[r + 5 * a.ts].x;
    }
#pragma unroll
    for (int i = 0; i < HALF; ++i) {
      const int j = h0 + i, row = t + T * j;
      const int64_t r = (int64_t)row * inner;
      float2 nv = v[j];
      if (KIND == FSM_NL_KS && (a.flags & FSM_FLAG_REMOVE_MEAN) && row == 0 && j0 == 0) nv = csub(nv, a.dc[0]);
      nv = cscale(nv, a.coef);
      if (srcp) nv = cadd(nv, srcp[r]);
      float2 tb[6];
      tb[0] = em[i];
      tb[1] = e2[i];
      tb[2] = make_float2(ca[i], 0.f);
      tb[3] = tb[4] = tb[5] = make_float2(cb[i], 0.f);
      float2 acc, q;
      const float2 st = setdrk4_pre<STG>(nv, o1[j], (STG == 1 || STG == 2) ? o2[i] : o1[j], tb, 1, acc, q);
      if (STG <= 2) accp[r] = acc;
      if (STG == 0) qp[r] = q;
      if (STG == 3) {
        up[r] = st;
        if (a.slot >= 0 && last) a.traj[(((int64_t)b * a.n_frames + a.slot) * C + cg) * S + r + j0] = st;
      }
      v[j] = st;
    }
  }
}

// N_s of a point's channels: the Leray projection, the KS batch mean, coefficient and source.
template <int NX, int KIND, int DIM>
__device__ __forceinline__ void axis0_nonlinear(const StepArgs& a, float2 (&nv)[RegKind<KIND, DIM>::CG], int b,
                                                int64_t j0, int row, int cg) {
  using K = RegKind<KIND, DIM>;
  constexpr int C = K::C, CG = K::CG;
  if (KIND == FSM_NL_LERAY) nv_leray<DIM, CG>(nv, point_k<DIM>(a, row, j0), row, j0, a, NX);
  if (KIND == FSM_NL_KS && (a.flags & FSM_FLAG_REMOVE_MEAN) && row == 0 && j0 == 0) nv[0] = csub(nv[0], a.dc[0]);
#pragma unroll
  for (int f = 0; f < CG; ++f) {
    nv[f] = cscale(nv[f], a.coef);
    if (a.src)
      nv[f] = cadd(nv[f], a.src[((int64_t)(a.src_batch > 1 ? b : 0) * C + cg * CG + f) * a.S +
                                (int64_t)row * (a.S / NX) + j0]);
  }
}

// The stage update of a thread's points, all channels of the group, in registers: SETDRK4 stage STG
// (INTEG FSM_SETDRK4), the right-hand side itself (FSM_APPLY), or the priming launch (STG -1), which
// only reads the state.
template <int NX, int KIND, int DIM, int INTEG, int STG>
__device__ __forceinline__ void axis0_update(const StepArgs& a, float2 (&v)[RegKind<KIND, DIM>::CG][RegShape<NX>::E],
                                             int b, int64_t j0, int t, int cg, bool last) {
  using K = RegKind<KIND, DIM>;
  constexpr int T = RegShape<NX>::T, E = RegShape<NX>::E, C = K::C, CG = K::CG;
  const int64_t S = a.S, inner = S / NX;
  float2* __restrict__ state = a.state;
  float2* __restrict__ aux = a.aux;
  float2* __restrict__ traj = a.traj;
  const float2* __restrict__ tab = a.tab;
#pragma unroll
  for (int i = 0; i < E; ++i) {
    const int row = t + T * i;
    const int64_t sidx = (int64_t)row * inner + j0;
    float2 nv[CG];
    if (STG >= 0) {
#pragma unroll
      for (int f = 0; f < CG; ++f) nv[f] = v[f][i];
      axis0_nonlinear<NX, KIND, DIM>(a, nv, b, j0, row, cg);
    }
#pragma unroll
    for (int f = 0; f < CG; ++f) {
      const int c = cg * CG + f;
      float2* up = state + ((int64_t)b * C + c) * S + sidx;
      const int64_t toff = (tab_batch(a, b) * a.lin_ch + (a.lin_ch > 1 ? c : 0)) * S + sidx;
      float2 st;
      if (STG < 0) {
        st = *up;
      } else if (INTEG == FSM_APPLY) {
        st = cfma(tab[toff], *up, nv[f]);
        *up = st;
      } else {
        float2* accp = aux + ((int64_t)b * a.n_aux * C + c) * S + sidx;
        float2* qp = aux + ((int64_t)b * a.n_aux * C + (a.n_aux > 1 ? C : 0) + c) * S + sidx;
        st = etd_stage_c<INTEG, STG>(nv[f], up, accp, qp, tab + toff, a.ts);
      }
      if (a.slot >= 0 && (STG < 0 || last)) traj[(((int64_t)b * a.n_frames + a.slot) * C + c) * S + sidx] = st;
      v[f][i] = st;
    }
  }
}

// The stage update of the other schemes, dispatched at run time: one rolled loop over the thread's
// points, which pass through its own words of the shared buffer x (unrolled over registers the
// dispatch would be repeated for every point).
template <int NX, int KIND, int DIM>
__device__ __forceinline__ void axis0_update_any(const StepArgs& a, float2 (&v)[RegKind<KIND, DIM>::CG][RegShape<NX>::E],
                                                 float2* __restrict__ x, int b, int64_t j0, int t, int cg, bool last) {
  using K = RegKind<KIND, DIM>;
  constexpr int T = RegShape<NX>::T, E = RegShape<NX>::E, C = K::C, CG = K::CG;
  const int64_t S = a.S, inner = S / NX;
  // (a channel at a time would need the Leray projection's other channels: the group's go together)
  float2* xs = x + threadIdx.x;
#pragma unroll
  for (int f = 0; f < CG; ++f)
#pragma unroll
    for (int i = 0; i < E; ++i) xs[(f * E + i) * 256] = v[f][i];
#pragma unroll 1
  for (int i = 0; i < E; ++i) {
    const int row = t + T * i;
    const int64_t sidx = (int64_t)row * inner + j0;
    float2 nv[CG];
#pragma unroll
    for (int f = 0; f < CG; ++f) nv[f] = xs[(f * E + i) * 256];
    axis0_nonlinear<NX, KIND, DIM>(a, nv, b, j0, row, cg);
#pragma unroll
    for (int f = 0; f < CG; ++f) {
      const int c = cg * CG + f;
      float2* accp = a.aux + ((int64_t)b * a.n_aux * C + c) * S + sidx;
      float2* qp = a.aux + ((int64_t)b * a.n_aux * C + (a.n_aux > 1 ? C : 0) + c) * S + sidx;
      const int64_t toff = (tab_batch(a, b) * a.lin_ch + (a.lin_ch > 1 ? c : 0)) * S + sidx;
      const float2 st = etd_stage(a.integ, a.stage, nv[f], a.state + ((int64_t)b * C + c) * S + sidx, accp, qp,
                                  a.tab + toff, a.ts, (int64_t)C * S);
      if (a.slot >= 0 && last) a.traj[(((int64_t)b * a.n_frames + a.slot) * C + c) * S + sidx] = st;
      xs[(f * E + i) * 256] = st;
    }
  }
#pragma unroll
  for (int f = 0; f < CG; ++f)
#pragma unroll
    for (int i = 0; i < E; ++i) v[f][i] = xs[(f * E + i) * 256];
}

// Axis-0 pass (2D: the column pass; 3D: the x pass). A CTA owns W adjacent inner columns (contiguous
// in memory) of one sample, all NX rows, a column's points in the registers of its T threads
// throughout (col_fft):
//   1. forward transform along axis 0 of the products -> N (+ Leray projection, + source)
//   2. stage update at every point, recording when a step completes
//   3. next stage field (mask, 1/N, i kx, streamfunction) -> inverse transform -> mid fields
// FAST: a SETDRK4 stage launch of a program with channel groups of one channel (the hoisted update,
// k_axis0_r2); otherwise any scheme, the priming launch included (k_axis0_r). STG: the stage of a FAST launch where the kernel has one of its own
// (-1: read from the arguments, the multi-plan kernels). PRIME: the priming launch alone (no transform of
// products, no other update compiled in).
// The code of a launch is kept small (one stage's update, one copy of the inverse transform).
// One channel group cg: a CTA of its own per group, so that the channels of a velocity run
// side by side instead of one after the other (3D Burgers 64^3 x 3: the x pass had 198 CTAs of three
// channels each; with the kept columns of the 3D passes 7.03 -> 5.60 ms per 20 steps).
// Bound: the latency of its rounds of loads (L2 hits: 6 of 12 cycles per issue at two CTAs per SM on
// 256^2 x 34) and instruction issue. Against the staged tiles it replaced (products, update and each
// field through shared tiles, tables loaded as used): vorticity 256^2 x 64 9.45 -> 8.68 ms per 50
// steps, 512^2 x 5 6.86 -> 6.37 ms per 40, 3D Burgers 256^3 17.0 -> 14.3 ms per 4, 64^3 x 3 5.62 ->
// 5.06 ms per 20.
template <int NX, int KIND, int DIM, bool FAST, int STG = -1, bool PRIME = false>
__device__ __forceinline__ void axis0_body(const StepArgs& a, int tile, int b, int cg) {
  using Cfg = ColCfg<NX>;
  using K = RegKind<KIND, DIM>;
  constexpr int T = Cfg::T, E = Cfg::E, W = Cfg::W, C = K::C, CG = K::CG;
  extern __shared__ float2 smem[];
  float2* twt = smem;       // NX
  float* kxs = (float*)(smem + NX);     // NX
  float2* buf = smem + NX + NX / 2;     // two exchange buffers
  int par = 0;
  const int g = threadIdx.x % W, t = threadIdx.x / W;
  const int64_t c0 = (int64_t)tile * W;
  const int64_t S = a.S, inner = S / NX;
  const bool in = c0 + g < inner;
  const int64_t j0 = in ? c0 + g : inner - 1;  // threads beyond the last column repeat it and store nothing
  load_reg_twiddles<NX>(twt, a.tw, threadIdx.x, 256);
  for (int x = threadIdx.x; x < NX; x += 256) kxs[x] = a.kx[x];
  pdl_wait();
  const bool last = a.stage == a.nstages - 1;

  float2 st[CG][E];
  float2 o1[FAST ? E : 1];
  if (!PRIME && a.stage >= 0) {
#pragma unroll
    for (int f = 0; f < CG; ++f) {
      const float2* src = a.prod + ((int64_t)b * a.n_prod + cg * CG + f) * a.ms + j0;
#pragma unroll
      for (int j = 0; j < E; ++j) st[f][j] = src[(int64_t)(t + T * j) * a.wp];
    }
    if constexpr (FAST) {
      const float2* o = ((STG >= 0 ? STG : a.stage) <= 1 ? a.state + ((int64_t)b * C + cg) * S : a.aux + ((int64_t)b * a.n_aux * C + cg) * S) + j0;
#pragma unroll
      for (int j = 0; j < E; ++j) o1[j] = o[(int64_t)(t + T * j) * inner];
    }
    __syncthreads();  // the twiddles and wavenumbers
#pragma unroll
    for (int f = 0; f < CG; ++f) col_fft<NX, false>(st[f], buf, par, twt, t, g);
  } else {
    __syncthreads();
  }
  if (in) {
    if constexpr (PRIME) {
      axis0_update<NX, KIND, DIM, -1, -1>(a, st, b, j0, t, cg, last);
    } else if constexpr (FAST && STG >= 0) {
      axis0_update_hoisted<NX, KIND, DIM, (STG >= 0 ? STG : 0)>(a, st[0], o1, b, j0, t, cg, last);
    } else if constexpr (FAST) {
      switch (a.stage) {
        case 0: axis0_update_hoisted<NX, KIND, DIM, 0>(a, st[0], o1, b, j0, t, cg, last); break;
        case 1: axis0_update_hoisted<NX, KIND, DIM, 1>(a, st[0], o1, b, j0, t, cg, last); break;
        case 2: axis0_update_hoisted<NX, KIND, DIM, 2>(a, st[0], o1, b, j0, t, cg, last); break;
        default: axis0_update_hoisted<NX, KIND, DIM, 3>(a, st[0], o1, b, j0, t, cg, last); break;
      }
    } else if (CG > 1 && a.stage >= 0 && a.integ == FSM_SETDRK4) {
      switch (a.stage) {
        case 0: axis0_update<NX, KIND, DIM, FSM_SETDRK4, 0>(a, st, b, j0, t, cg, last); break;
        case 1: axis0_update<NX, KIND, DIM, FSM_SETDRK4, 1>(a, st, b, j0, t, cg, last); break;
        case 2: axis0_update<NX, KIND, DIM, FSM_SETDRK4, 2>(a, st, b, j0, t, cg, last); break;
        default: axis0_update<NX, KIND, DIM, FSM_SETDRK4, 3>(a, st, b, j0, t, cg, last); break;
      }
    } else if (a.stage < 0) {
      axis0_update<NX, KIND, DIM, -1, -1>(a, st, b, j0, t, cg, last);
    } else if (a.integ == FSM_APPLY) {
      axis0_update<NX, KIND, DIM, FSM_APPLY, 0>(a, st, b, j0, t, cg, last);
    } else {
      // words of its own in a buffer of its own (behind the exchange buffers)
      axis0_update_any<NX, KIND, DIM>(a, st, smem + Cfg::WORDS, b, j0, t, cg, last);
    }
  }
  pdl_trigger();
  if (!a.emit) return;  // uniform
  // 2D: columns from hk on are dealiased and the row pass does not read them: nothing to store.
  // 3D: the next passes read the columns (jm, jl) with jm kept and jl < hk.
  if (DIM == 2 && c0 >= (int64_t)a.hk) return;  // uniform
  bool live = in;
  if (DIM == 2) live = j0 < (int64_t)a.hk && in;
  else if (live) live = (int)(j0 % a.H) < a.hk && (a.hk == a.H || a.keepm[(int)(j0 / a.H)]);
  if (a.tile_zero && a.tile_zero[tile]) {
    if (DIM == 3 && a.hk < a.H) return;
    // every column of this tile is dealiased: the next-stage fields are zero here
    constexpr int NMO = (KIND == FSM_NL_CONVECTION) ? 2 : K::NMG;  // fields of this channel group
    const int m0 = (KIND == FSM_NL_CONVECTION) ? cg * 2 : 0;
#pragma unroll 1
    for (int mf = 0; mf < NMO; ++mf) {
      float2* dst = a.mid + ((int64_t)b * a.n_mid + m0 + mf) * a.ms + j0;
#pragma unroll
      for (int j = 0; j < E; ++j)
        if (live) dst[(int64_t)(t + T * j) * a.wp] = make_float2(0.f, 0.f);
    }
    return;  // uniform across the CTA
  }
  const PointK<DIM> gk = point_k<DIM>(a, 0, j0);
  const uint8_t kc = (DIM == 2) ? a.keepy[j0] : (uint8_t)(a.keepm[(int)(j0 / a.H)] & a.keepy[(int)(j0 % a.H)]);
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const int row = t + T * j;
    const float m = (float)(a.keepx[row] & kc) * a.scale;
#pragma unroll
    for (int f = 0; f < CG; ++f) st[f][j] = cscale(st[f][j], m);
  }
  // The streamfunction's 1 / lap, once a point: fast division up to 256 points (within 2 ulp for |lap| below
  // 2^126, far above any mesh's 2 (pi NX / L)^2), rounded at 512 points, as those grids always had it. Once
  // a field, rounded: vorticity 512^2 x 5 5.21 ms per 40 steps; once a point: 4.76 (4.79 with the fast
  // division once a field; 256^2 x 64 8.29 -> 7.96 ms per 50).
  constexpr bool exact = NX == 512;
  // (channel by channel for the Leray projection's groups: the fields of channel f are 2 f, 2 f + 1)
#pragma unroll
  for (int f = 0; f < CG; ++f) {
#pragma unroll 1
  for (int i = f * 2; i < (CG > 1 ? f * 2 + 2 : K::NMG); ++i) {
    // vorticity: 0: psi = -w/lap, 1: i kx psi, 2: w, 3: i kx w, the fields of w first and psi in w's place
    // then; KS: 0: phi, 1: i kx phi; velocity (per channel): u_c, i kx u_c
    const int mf = KIND == FSM_NL_VORTICITY ? (i + 2) & 3 : i;
    if (KIND == FSM_NL_VORTICITY && mf == 0) {
#pragma unroll
      for (int j = 0; j < E; ++j) {
        const float kxv = kxs[t + T * j];
        const float lap = -(kxv * kxv + gk.ky * gk.ky);
        const float il = (lap == 0.f) ? 1.f : exact ? 1.f / lap : __fdividef(1.f, lap);
        st[f][j] = cscale(st[f][j], -il);
      }
    }
    float2 v[E];
#pragma unroll
    for (int j = 0; j < E; ++j) {
      const float2 ix = cscale(cmuli(st[f][j]), kxs[t + T * j]);
      v[j] = (mf & 1) ? ix : st[f][j];
    }
    col_fft<NX, true>(v, buf, par, twt, t, g);
    const int mout = (KIND == FSM_NL_CONVECTION) ? cg * 2 + mf : mf;
    float2* dst = a.mid + ((int64_t)b * a.n_mid + mout) * a.ms + j0;
    if (live) {
#pragma unroll
      for (int j = 0; j < E; ++j) dst[(int64_t)(t + T * j) * a.wp] = v[j];
    }
  }
  }
}

template <int NY>
struct RowCfgR {
  using RS = RegShape<NY>;
  static constexpr int T = RS::T;
  static constexpr int E = RS::E;
  static constexpr int SCR = reg_scratch<NY>();
};

__device__ __forceinline__ float2 herm_z(float2 A, float2 B, bool selfc, bool hi) {
  if (selfc) {
    A.y = 0.f;
    B.y = 0.f;
  }
  if (hi) {
    A.y = -A.y;
    B.y = -B.y;
  }
  return make_float2(A.x - B.y, A.y + B.x);  // A + i B
}

// Split the transform of p0 + i p1 (lane t holds K = t + T j in register j)
// into the half spectra of p0 and p1 and store k = 0..NY/2.
template <int NY>
__device__ __forceinline__ void split_store_r(const float2 (&zp)[RegShape<NY>::E], int t, int lane,
                                              float2* __restrict__ out0, float2* __restrict__ out1) {
  constexpr int T = RegShape<NY>::T, E = RegShape<NY>::E;
  constexpr int J = NY / (2 * T);
  const int partner_lane = (lane & ~(T - 1)) | ((T - t) & (T - 1));
#pragma unroll
  for (int j = 0; j <= J; ++j) {
    const float2 send = zp[E - 1 - j];
    float2 recv;
    recv.x = __shfl_sync(0xffffffffu, send.x, partner_lane);
    recv.y = __shfl_sync(0xffffffffu, send.y, partner_lane);
    const float2 partner = (t == 0) ? zp[(E - j) & (E - 1)] : recv;
    const int k = t + T * j;
    if (k <= NY / 2) {
      const float2 zm = cconj(partner);
      out0[k] = cscale(cadd(zp[j], zm), 0.5f);
      out1[k] = cscale(cmulmi(csub(zp[j], zm)), 0.5f);
    }
  }
}

// HK: the stage fields' stored columns (FsmPlan::hk), NY/2 + 1 when every column is stored.
template <int NY, int KIND, int HK>
__device__ __forceinline__ void plane_row_body(const StepArgs& a, int blk, int b) {
  using Cfg = RowCfgR<NY>;
  constexpr int T = Cfg::T, E = Cfg::E, SCR = Cfg::SCR;
  extern __shared__ float2 smem[];
  float2* twt = smem;
  const int lane = threadIdx.x & 31;
  const int g = threadIdx.x / T, t = threadIdx.x % T;
  const int groups = blockDim.x / T;
  float2* scr = smem + NY + g * SCR;
  load_reg_twiddles<NY>(twt, a.tw, threadIdx.x, blockDim.x);
  pdl_wait();
  __syncthreads();
  const int r0 = (blk * groups + g) * 2;
  const int64_t S = a.ms;  // field stride of the stage fields and products
  const int64_t WP = a.wp;  // their row pitch
  const float* ky = a.ky;
  const float2* mid = a.mid + (int64_t)b * a.n_mid * S;
  float2* prod = a.prod + (int64_t)b * a.n_prod * S;

  const float2 zero = make_float2(0.f, 0.f);
  if (KIND == FSM_NL_VORTICITY || KIND == FSM_NL_KS) {
    float p[2][E];
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      const int64_t roff = (int64_t)(r0 + rr) * WP;
      float2 Z1[E], Z2[E];
#pragma unroll
      for (int j = 0; j < E; ++j) {
        if (reg_dead<NY, T, HK>(j)) {
          Z1[j] = zero;
          Z2[j] = zero;
          continue;
        }
        const int k = t + T * j;
        const bool hi = k > NY / 2;
        const int kk = hi ? NY - k : k;
        const bool selfc = (kk == 0) || (kk == NY / 2);
        const bool live = HK > NY / 2 || kk < HK;
        const float kyv = ky[kk];
        if (KIND == FSM_NL_VORTICITY) {
          const float2 m0 = live ? mid[roff + kk] : zero, m1 = live ? mid[S + roff + kk] : zero;
          const float2 m2 = live ? mid[2 * S + roff + kk] : zero, m3 = live ? mid[3 * S + roff + kk] : zero;
          // u_x + i u_y with u_x <- i ky psi, u_y <- -(i kx psi); w_x + i w_y with w_x <- i kx w, w_y <- i ky w
          Z1[j] = herm_z(cscale(cmuli(m0), kyv), make_float2(-m1.x, -m1.y), selfc, hi);
          Z2[j] = herm_z(m3, cscale(cmuli(m2), kyv), selfc, hi);
        } else {
          const float2 m0 = live ? mid[roff + kk] : zero, m1 = live ? mid[S + roff + kk] : zero;
          Z1[j] = herm_z(m1, cscale(cmuli(m0), kyv), selfc, hi);  // phi_x + i phi_y
        }
      }
      reg_fft<NY, true>(Z1, scr, twt, t);
      if (KIND == FSM_NL_VORTICITY) {
        reg_fft<NY, true>(Z2, scr, twt, t);
#pragma unroll
        for (int j = 0; j < E; ++j) p[rr][j] = Z1[j].x * Z2[j].x + Z1[j].y * Z2[j].y;
      } else {
#pragma unroll
        for (int j = 0; j < E; ++j) p[rr][j] = 0.5f * (Z1[j].x * Z1[j].x + Z1[j].y * Z1[j].y);
      }
    }
    float2 zp[E];
#pragma unroll
    for (int j = 0; j < E; ++j) zp[j] = make_float2(p[0][j], p[1][j]);
    pdl_trigger();
    reg_fft<NY, false>(zp, scr, twt, t);
    split_store_r<NY>(zp, t, lane, prod + (int64_t)r0 * WP, prod + (int64_t)(r0 + 1) * WP);
  } else {
    // convection, C = 2: conv_c = u0 dx u_c + u1 dy u_c
#pragma unroll 1
    for (int rr = 0; rr < 2; ++rr) {
      const int64_t roff = (int64_t)(r0 + rr) * WP;
      float2 Z1[E], Z2[E];
#pragma unroll
      for (int j = 0; j < E; ++j) {
        if (reg_dead<NY, T, HK>(j)) {
          Z1[j] = zero;
          Z2[j] = zero;
          continue;
        }
        const int k = t + T * j;
        const bool hi = k > NY / 2;
        const int kk = hi ? NY - k : k;
        const bool selfc = (kk == 0) || (kk == NY / 2);
        const bool live = HK > NY / 2 || kk < HK;
        Z1[j] = live ? herm_z(mid[roff + kk], mid[2 * S + roff + kk], selfc, hi) : zero;       // u0 + i u1
        Z2[j] = live ? herm_z(mid[S + roff + kk], mid[3 * S + roff + kk], selfc, hi) : zero;   // dx u0 + i dx u1
      }
      reg_fft<NY, true>(Z1, scr, twt, t);
      reg_fft<NY, true>(Z2, scr, twt, t);
      float2 acc[E];
      float u1[E];
#pragma unroll
      for (int j = 0; j < E; ++j) {
        acc[j] = make_float2(Z1[j].x * Z2[j].x, Z1[j].x * Z2[j].y);
        u1[j] = Z1[j].y;
      }
#pragma unroll
      for (int j = 0; j < E; ++j) {
        if (reg_dead<NY, T, HK>(j)) {
          Z2[j] = zero;
          continue;
        }
        const int k = t + T * j;
        const bool hi = k > NY / 2;
        const int kk = hi ? NY - k : k;
        const bool selfc = (kk == 0) || (kk == NY / 2);
        const bool live = HK > NY / 2 || kk < HK;
        const float kyv = ky[kk];
        Z2[j] = live ? herm_z(cscale(cmuli(mid[roff + kk]), kyv), cscale(cmuli(mid[2 * S + roff + kk]), kyv), selfc, hi)
                     : zero;
      }
      reg_fft<NY, true>(Z2, scr, twt, t);  // dy u0 + i dy u1
#pragma unroll
      for (int j = 0; j < E; ++j) {
        acc[j].x += u1[j] * Z2[j].x;
        acc[j].y += u1[j] * Z2[j].y;
      }
      if (rr == 1) pdl_trigger();
      reg_fft<NY, false>(acc, scr, twt, t);
      split_store_r<NY>(acc, t, lane, prod + roff, prod + S + roff);
    }
  }
}

}  // namespace fsm
