// Fused 1D integration: a group of T threads per sample runs every step and stage of the
// exponential Runge-Kutta scheme with the state and the scheme's running sums resident in shared
// memory, and writes recorded frames straight into the trajectory. One launch per integrate call.
//
// Nonlinear terms (input dealiased, output not, operator/_base.py:375-403):
//  FSM_NL_CONVECTION  u u_x: one inverse complex FFT of Z = D + i G with
//                     D = mask*u_hat/N and G = i k D gives z = u + i u_x
//                     (operator/generic/_convection.py:43-46);
//  FSM_NL_KS          0.5 u_x^2 (operator/dedicated/_ks_convection.py:27-38).
// followed by one forward FFT of the real product.
//
// Transforms. Thread t keeps the elements t + T j (j < E) in registers from the spectral update
// through the inverse transform, the product and the forward transform back to the update: the
// first and the last pass of a transform have radix E, whose inputs and outputs are exactly those
// elements. Between passes the group exchanges through one of two shared buffers in turn, so an
// exchange costs one barrier (a buffer is written again only after the other one's barrier). The
// thread that holds mode k < N/2 updates it and hands the conjugate mode N - k to its owner.
// Bound: the latency of the chain of passes and exchanges of one sample (a few warps per SM);
// the transforms ran through shared memory in every pass before, with two barriers each.
// Measured, us per stage (before -> now): 128 points
// 1.54 -> 0.57, 256: 2.23 -> 0.76, 1024: 5.3 -> 1.15, 2048: 5.1 -> 1.9, 4096: 10.2 -> 2.9 (1 to 32 samples).
#include "fsm_internal.cuh"
#include "fsm_linefft.cuh"

namespace fsm {

// The inverse transform's inputs from the stage field `a` at mode k <= N/2: the value at k and, for
// 0 < k < N/2, the one at N - k.
template <int N, int KIND>
__device__ __forceinline__ float2 line_build(int k, float2 a, float mask, float kxv, float2* mirror) {
  const float2 d = cscale(a, mask);
  float2 G = make_float2(-kxv * d.y, kxv * d.x);  // i k d
  const bool selfc = (k == 0) || (k == N / 2);
  if (selfc) G.y = 0.f;
  if (KIND == FSM_NL_CONVECTION) {
    float2 D = d;
    if (selfc) D.y = 0.f;
    *mirror = make_float2(D.x + G.y, G.x - D.y);
    return make_float2(D.x - G.y, D.y + G.x);
  } else {  // FSM_NL_KS
    *mirror = cconj(G);
    return G;
  }
}

// One sample's integration by the T threads of its sub-group (`lane_on`; spare lanes of a short
// sample only keep the barriers or repeat): the twiddles `tw` are in shared memory already (visible after the body's first
// barrier); `reg` is the sample's shared-memory region. `active` false runs the body on the data of
// a valid sample without writing global memory (spare sub-groups of a k_line_multi CTA).
template <int N, int KIND, bool REGS>
__device__ __forceinline__ void line_body(const StepArgs& a, int b, int t, int id, const float2* __restrict__ tw,
                                          float2* reg, bool lane_on, bool active) {
  using Cfg = LineCfg<N>;
  // with everything in registers the lanes beyond T repeat the work of lane t % T (same values to the
  // same shared words) instead of branching around it; they write nothing global
  const bool on = REGS || lane_on;
  constexpr int H = Cfg::H, T = Cfg::T, E = Cfg::E;
  constexpr int M = E / 2 + 1;  // modes t + T j, j < M (the last one, N/2, is thread 0's)
  // the buffers alternate over the exchanges of a stage: two transforms and the conjugate modes
  constexpr int XF = line_exchanges<N>();
  // A transform of up to 64 points takes T < 32 lanes with M modes each. The schemes dispatched at run time
  // (REGS false) spread the modes over the whole warp for their update, through the exchange buffers: M updates one
  // after the other cost more than the exchange (RK4 of one sample, 40 steps, us: 16 points 185 -> 115, 32: 201 -> 134, 64:
  // 214 -> 166).
  constexpr bool SPREAD = !REGS && T < 32;
  constexpr int MW = (H + 31) / 32;  // modes of a lane then
  const int lane = threadIdx.x & 31;
  float2* u = reg + 2 * Cfg::NB;
  float2* acc = u + H;  // running sums: acc, q (Runge-Kutta: n_aux arrays H apart)
  float2* q = acc + H;
  float2* gstate = a.state + (int64_t)b * H;
  const int64_t toff = tab_batch(a, b) * H;
  const float2* tab = a.tab + toff;
  const float2* src = a.src ? a.src + (int64_t)(a.src_batch > 1 ? b : 0) * H : nullptr;
  const int slot0 = a.slots ? a.slots[0] : -1;
  const bool dc = KIND == FSM_NL_KS && (a.flags & FSM_FLAG_REMOVE_MEAN) && active && lane_on && t == 0;
  float2 v[E];
  float kxr[M], mask[M];
  // REGS: the state (between stages 0 and 1 exp(dt L / 2) u), the running sums and the tables
  float2 ru[REGS ? M : 1], racc[REGS ? M : 1], rq[REGS ? M : 1], tE[REGS ? M : 1], tE2[REGS ? M : 1];
  float tc[4][REGS ? M : 1];  // c1, c4, c5, c6
  int par = 0;  // the buffer of the next exchange

  // stage field at the thread's modes (registers x) -> inverse transform inputs in v
  auto emit = [&](const float2 (&x)[M]) {
    float2* ex = reg + par * Cfg::NB;
    par ^= 1;
    if (on) {
#pragma unroll
      for (int j = 0; j < M; ++j) {
        const int k = t + T * j;
        if (j == M - 1 && t != 0) break;
        float2 mir;
        const float2 z = line_build<N, KIND>(k, x[j], mask[j], kxr[j], &mir);
        if (k > 0 && k < N / 2) ex[line_pad(N - k)] = mir;
        if (j < M - 1) v[j] = z;
        else ex[line_pad(k)] = z;
      }
    }
    line_sync<N>(id);
    if (on) {
#pragma unroll
      for (int j = E / 2; j < E; ++j) v[j] = ex[line_pad(t + T * j)];
    }
  };

  float skx[SPREAD ? MW : 1], smask[SPREAD ? MW : 1];
  if constexpr (SPREAD) {
#pragma unroll
    for (int r = 0; r < MW; ++r) {
      const int k = min(lane + 32 * r, N / 2);
      skx[r] = a.kx[k];
      smask[r] = (float)a.keepx[k] * a.scale;
    }
  }
  float2 x[M];
  if (on) {
#pragma unroll
    for (int j = 0; j < M; ++j) {
      if (j == M - 1 && t != 0) break;
      const int k = t + T * j;
      x[j] = gstate[k];
      kxr[j] = a.kx[k];
      mask[j] = (float)a.keepx[k] * a.scale;
      if constexpr (REGS) {
        ru[j] = x[j];
        tE[j] = tab[k];
        tE2[j] = tab[a.ts + k];
        // the SETDRK coefficients are real (k_phi_tables)
        tc[0][j] = tab[2 * a.ts + k].x;
        tc[1][j] = tab[3 * a.ts + k].x;
        tc[2][j] = tab[4 * a.ts + k].x;
        tc[3][j] = tab[5 * a.ts + k].x;
      } else {
        u[k] = x[j];
      }
      if (slot0 >= 0 && active && lane_on) a.traj[((int64_t)b * a.n_frames + slot0) * H + k] = x[j];
    }
  }
  if (dc) a.dc[(int64_t)a.steps * a.nstages * a.B + b] = x[0];  // initial k = 0 value
  if (a.steps > 0) emit(x);
  const int ns = a.nstages;
#pragma unroll 1
  for (int step = 0; step < a.steps; ++step) {
#pragma unroll 1
    for (int s = 0; s < ns; ++s) {
      line_passes<N, true, 1>(v, reg + par * Cfg::NB, reg + (par ^ 1) * Cfg::NB, tw, t, id, on);
      par ^= XF & 1;
#pragma unroll
      for (int j = 0; j < E; ++j) {
        const float p = (KIND == FSM_NL_CONVECTION) ? v[j].x * v[j].y : 0.5f * v[j].x * v[j].x;
        v[j] = make_float2(p, 0.f);
      }
      line_passes<N, false, 1>(v, reg + par * Cfg::NB, reg + (par ^ 1) * Cfg::NB, tw, t, id, on);
      par ^= XF & 1;
      const bool last = (s == ns - 1);
      const int slot = (last && a.slots) ? a.slots[step + 1] : -1;
      // k = 0 of the product, for the batch-mean fix-up (k_line_dc_fixup)
      if (dc) a.dc[((int64_t)step * ns + s) * a.B + b] = v[0];
      if constexpr (SPREAD) {
        float2* ex = reg + par * Cfg::NB;
        float2* zx = reg + (par ^ 1) * Cfg::NB;
        if (on) {
#pragma unroll
          for (int j = 0; j < M; ++j) {
            if (j == M - 1 && t != 0) break;
            ex[line_pad(t + T * j)] = v[j];
          }
        }
        line_sync<N>(id);
#pragma unroll
        for (int r = 0; r < MW; ++r) {
          const int k = lane + 32 * r;
          if (k < H) {
            float2 nv = cscale(ex[line_pad(k)], a.coef);
            if (src) nv = cadd(nv, src[k]);
            const float2 xk = etd_stage(a.integ, s, nv, u + k, acc + k, q + k, tab + k, a.ts, H);
            if (slot >= 0 && active) a.traj[((int64_t)b * a.n_frames + slot) * H + k] = xk;
            float2 mir;
            zx[line_pad(k)] = line_build<N, KIND>(k, xk, smask[r], skx[r], &mir);
            if (k > 0 && k < N / 2) zx[line_pad(N - k)] = mir;
          }
        }
        line_sync<N>(id);
        if (on) {
#pragma unroll
          for (int j = 0; j < E; ++j) v[j] = zx[line_pad(t + T * j)];
        }
        continue;
      }
      if (on) {
#pragma unroll
        for (int j = 0; j < M; ++j) {
          x[j] = cscale(v[j], a.coef);
          if (src && (j < M - 1 || t == 0)) x[j] = cadd(x[j], src[t + T * j]);
        }
        if constexpr (REGS) {
          // the recurrences of etd_stage_c<FSM_SETDRK4, s>
#pragma unroll
          for (int j = 0; j < M; ++j) {
            const float2 nv = x[j];
            const float2 c1 = make_float2(tc[0][j], 0.f);
            if (s == 0) {
              const float2 e2u = cexpmul(tE2[j], ru[j]);
              x[j] = cfma(c1, nv, e2u);
              racc[j] = cfma(make_float2(tc[1][j], 0.f), nv, cexpmul(tE[j], ru[j]));
              rq[j] = cfma(make_float2(-c1.x, -c1.y), nv, cexpmul(tE2[j], x[j]));
              ru[j] = e2u;
            } else if (s == 1) {
              racc[j] = cfma(make_float2(2.f * tc[2][j], 0.f), nv, racc[j]);
              x[j] = cfma(c1, nv, ru[j]);
            } else if (s == 2) {
              racc[j] = cfma(make_float2(2.f * tc[2][j], 0.f), nv, racc[j]);
              x[j] = cfma(cscale(c1, 2.f), nv, rq[j]);
            } else {
              x[j] = cfma(make_float2(tc[3][j], 0.f), nv, racc[j]);
              ru[j] = x[j];
            }
          }
        } else {
          auto stage = [&](auto&& f) {
#pragma unroll
            for (int j = 0; j < M; ++j) {
              if (j == M - 1 && t != 0) break;
              const int k = t + T * j;
              x[j] = f(x[j], u + k, acc + k, q + k, tab + k);
            }
          };
          using F2 = float2;
          if (E > 8 && a.integ == FSM_SETDRK4) {
            switch (s) {
              case 0: stage([&](F2 n, F2* pu, F2* pa, F2* pq, const F2* pt) { return etd_stage_c<FSM_SETDRK4, 0>(n, pu, pa, pq, pt, a.ts); }); break;
              case 1: stage([&](F2 n, F2* pu, F2* pa, F2* pq, const F2* pt) { return etd_stage_c<FSM_SETDRK4, 1>(n, pu, pa, pq, pt, a.ts); }); break;
              case 2: stage([&](F2 n, F2* pu, F2* pa, F2* pq, const F2* pt) { return etd_stage_c<FSM_SETDRK4, 2>(n, pu, pa, pq, pt, a.ts); }); break;
              default: stage([&](F2 n, F2* pu, F2* pa, F2* pq, const F2* pt) { return etd_stage_c<FSM_SETDRK4, 3>(n, pu, pa, pq, pt, a.ts); }); break;
            }
          } else {
            stage([&](F2 n, F2* pu, F2* pa, F2* pq, const F2* pt) { return etd_stage(a.integ, s, n, pu, pa, pq, pt, a.ts, H); });
          }
        }
        if (slot >= 0 && active && lane_on) {
#pragma unroll
          for (int j = 0; j < M; ++j) {
            if (j == M - 1 && t != 0) break;
            const int k = t + T * j;
            a.traj[((int64_t)b * a.n_frames + slot) * H + k] = x[j];
          }
        }
      }
      if (!(last && step == a.steps - 1)) emit(x);
    }
  }
  if (lane_on && active) {
#pragma unroll
    for (int j = 0; j < M; ++j) {
      if (j == M - 1 && t != 0) break;
      gstate[t + T * j] = REGS ? ru[REGS ? j : 0] : u[t + T * j];
    }
  }
}

template <int N, int KIND, bool REGS>
__global__ void __launch_bounds__(LineCfg<N>::G) k_line(StepArgs a) {
  using Cfg = LineCfg<N>;
  extern __shared__ float2 smem[];
  line_twiddles<N>(smem, a.tw, threadIdx.x, Cfg::G);
  __syncthreads();
  line_body<N, KIND, REGS>(a, blockIdx.x, threadIdx.x % Cfg::T, 0, smem, smem + Cfg::TW, threadIdx.x < Cfg::T, true);
}

// Serving: the lines of several plans (one per grid size) advanced by one launch. CTAs
// [cta0[j], cta0[j + 1]) belong to plan j; each holds kLineMultiThreads / G samples of its plan,
// one per sub-group of G threads, with the twiddles shared and a region per sample.
template <int N>
struct LineMultiCfg {
  static constexpr int G = LineCfg<N>::G;
  static constexpr int P = kLineMultiThreads / G;  // samples per CTA
  static size_t smem(int n_aux) { return (LineCfg<N>::TW + P * LineCfg<N>::region(n_aux)) * sizeof(float2); }
};

template <int N, int KIND, bool REGS>
__device__ __forceinline__ void line_multi_cta(const StepArgs& a, int cta) {
  using Cfg = LineMultiCfg<N>;
  extern __shared__ float2 smem[];
  line_twiddles<N>(smem, a.tw, threadIdx.x, kLineMultiThreads);
  __syncthreads();
  const int sub = threadIdx.x / Cfg::G, t = threadIdx.x % Cfg::G;
  const int b = cta * Cfg::P + sub;
  const bool active = b < a.B;
  float2* reg = smem + LineCfg<N>::TW + (size_t)sub * LineCfg<N>::region(a.n_aux);
  line_body<N, KIND, REGS && LineCfg<N>::E <= 8>(a, active ? b : a.B - 1, t, sub + 1, smem, reg, t < LineCfg<N>::T, active);
}

template <int KIND, bool REGS>
__global__ void __launch_bounds__(kLineMultiThreads) k_line_multi(const __grid_constant__ LineMulti m) {
  int j = 0;
  while (j + 1 < m.count && (int)blockIdx.x >= m.cta0[j + 1]) ++j;
  const int cta = (int)blockIdx.x - m.cta0[j];
  switch (m.n[j]) {
    case 256: line_multi_cta<256, KIND, REGS>(m.a[j], cta); break;
    case 512: line_multi_cta<512, KIND, REGS>(m.a[j], cta); break;
    case 1024: line_multi_cta<1024, KIND, REGS>(m.a[j], cta); break;
    case 2048: line_multi_cta<2048, KIND, REGS>(m.a[j], cta); break;
    case 4096: line_multi_cta<4096, KIND, REGS>(m.a[j], cta); break;
  }
}

template <int N>
static void line_multi_shape(int n_aux, int batch, size_t* smem, int* ctas) {
  using Cfg = LineMultiCfg<N>;
  *smem = Cfg::smem(n_aux);
  *ctas = (batch + Cfg::P - 1) / Cfg::P;
}

template <int N, int KIND, bool REGS>
static int launch_line_r(const StepArgs& a, cudaStream_t st) {
  using Cfg = LineCfg<N>;
  const size_t smem = (Cfg::TW + Cfg::region(a.n_aux)) * sizeof(float2);
  int rc = prep_smem(k_line<N, KIND, REGS>, smem);
  if (rc) return rc;
  k_line<N, KIND, REGS><<<a.B, Cfg::G, smem, st>>>(a);
  return cuda_check(cudaGetLastError(), "k_line");
}

// SETDRK4 keeps its state and tables in registers where a thread has few modes (E <= 8).
template <int N, int KIND>
static int launch_line_n(const StepArgs& a, cudaStream_t st) {
  if constexpr (LineCfg<N>::E <= 8) {
    if (a.integ == FSM_SETDRK4) return launch_line_r<N, KIND, true>(a, st);
  }
  return launch_line_r<N, KIND, false>(a, st);
}

template <int KIND>
static int launch_line_kind(int n, const StepArgs& a, cudaStream_t st) {
  switch (n) {
    case 16: return launch_line_n<16, KIND>(a, st);
    case 32: return launch_line_n<32, KIND>(a, st);
    case 64: return launch_line_n<64, KIND>(a, st);
    case 128: return launch_line_n<128, KIND>(a, st);
    case 256: return launch_line_n<256, KIND>(a, st);
    case 512: return launch_line_n<512, KIND>(a, st);
    case 1024: return launch_line_n<1024, KIND>(a, st);
    case 2048: return launch_line_n<2048, KIND>(a, st);
    case 4096: return launch_line_n<4096, KIND>(a, st);
  }
  return set_error(FSM_ERR_UNSUPPORTED, "1D: unsupported length " + std::to_string(n));
}

// KSConvection with the mean removed over a batch (operator/dedicated/_ks_convection.py:35-36:
// re.mean() spans the whole batch). The mean only changes the k = 0 value of the nonlinear
// term, and the k = 0 mode never feeds back into the product (it is a gradient), so the line
// kernel runs with the per-sample values and records every stage's k = 0 product P_b in
// dc[step][stage][b]. k_line_dc_mean reduces each (step, stage) row over the batch, in a fixed
// order, into dc[steps * stages * B + B + row]; k_line_dc_fixup then replays the k = 0
// recurrence of each sample with coef * (P_b - mean) + source, the same arithmetic as the line
// kernel, and overwrites k = 0 of the state and of the recorded frames.
__global__ void __launch_bounds__(256) k_line_dc_mean(StepArgs a) {
  __shared__ float2 red[256];
  const int row = blockIdx.x;
  const float2* P = a.dc + (int64_t)row * a.B;
  float2 sum = make_float2(0.f, 0.f);
  for (int i = threadIdx.x; i < a.B; i += 256) sum = cadd(sum, P[i]);
  red[threadIdx.x] = sum;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] = cadd(red[threadIdx.x], red[threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const float inv = 1.f / (float)a.B;
    a.dc[(int64_t)a.steps * a.nstages * a.B + a.B + row] = cscale(red[0], inv);
  }
}

__global__ void k_line_dc_fixup(StepArgs a) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= a.B) return;
  const int ns = a.nstages;
  const int H = a.H;
  const float2* mean = a.dc + (int64_t)a.steps * ns * a.B + a.B;
  float2 u = a.dc[(int64_t)a.steps * ns * a.B + b];
  float2 aux[6] = {};  // the scheme's running sums at k = 0
  const float2* tab = a.tab + tab_batch(a, b) * H;
  const float2 src0 = a.src ? a.src[(int64_t)(a.src_batch > 1 ? b : 0) * H] : make_float2(0.f, 0.f);
  for (int step = 0; step < a.steps; ++step) {
    for (int s = 0; s < ns; ++s) {
      const int64_t row = (int64_t)step * ns + s;
      const float2 nv = cadd(cscale(csub(a.dc[row * a.B + b], mean[row]), a.coef), src0);
      (void)etd_stage(a.integ, s, nv, &u, aux, aux + 1, tab, a.ts, 1);
    }
    const int slot = a.slots ? a.slots[step + 1] : -1;
    if (slot >= 0) a.traj[((int64_t)b * a.n_frames + slot) * H] = u;
  }
  a.state[(int64_t)b * H] = u;
}

template <int KIND, bool REGS>
static int launch_line_multi_k(const LineMulti& m, int total, size_t smem, cudaStream_t st) {
  int rc = prep_smem(k_line_multi<KIND, REGS>, smem);
  if (rc) return rc;
  k_line_multi<KIND, REGS><<<total, kLineMultiThreads, smem, st>>>(m);
  return cuda_check(cudaGetLastError(), "k_line_multi");
}

int launch_line_multi(LineMulti& m, int kind, cudaStream_t st) {
  if (m.count < 1 || m.count > kLineMultiMax) return set_error(FSM_ERR_INVALID, "line multi: plan count");
  size_t smem = 0;
  int total = 0;
  for (int j = 0; j < m.count; ++j) {
    size_t sm = 0;
    int ctas = 0;
    const int B = m.a[j].B, na = m.a[j].n_aux;
    if (B < 1) return set_error(FSM_ERR_INVALID, "line multi: empty plan entry");
    switch (m.n[j]) {
      case 256: line_multi_shape<256>(na, B, &sm, &ctas); break;
      case 512: line_multi_shape<512>(na, B, &sm, &ctas); break;
      case 1024: line_multi_shape<1024>(na, B, &sm, &ctas); break;
      case 2048: line_multi_shape<2048>(na, B, &sm, &ctas); break;
      case 4096: line_multi_shape<4096>(na, B, &sm, &ctas); break;
      default: return set_error(FSM_ERR_UNSUPPORTED, "line multi: lengths 256..4096 only");
    }
    m.cta0[j] = total;
    total += ctas;
    smem = sm > smem ? sm : smem;
  }
  m.cta0[m.count] = total;
  bool regs = true;
  for (int j = 0; j < m.count; ++j) regs = regs && m.a[j].integ == FSM_SETDRK4;
  if (kind == FSM_NL_KS)
    return regs ? launch_line_multi_k<FSM_NL_KS, true>(m, total, smem, st)
                : launch_line_multi_k<FSM_NL_KS, false>(m, total, smem, st);
  if (kind == FSM_NL_CONVECTION)
    return regs ? launch_line_multi_k<FSM_NL_CONVECTION, true>(m, total, smem, st)
                : launch_line_multi_k<FSM_NL_CONVECTION, false>(m, total, smem, st);
  return set_error(FSM_ERR_UNSUPPORTED, "line multi: unsupported nonlinear term");
}

int launch_line(const FsmPlan* p, const StepArgs& a, cudaStream_t st) {
  switch (p->nl) {
    case FSM_NL_CONVECTION: return launch_line_kind<FSM_NL_CONVECTION>(p->n[0], a, st);
    case FSM_NL_KS: {
      int rc = launch_line_kind<FSM_NL_KS>(p->n[0], a, st);
      if (rc || !(p->flags & FSM_FLAG_REMOVE_MEAN) || a.steps == 0) return rc;
      k_line_dc_mean<<<a.steps * a.nstages, 256, 0, st>>>(a);
      rc = cuda_check(cudaGetLastError(), "k_line_dc_mean");
      if (rc) return rc;
      k_line_dc_fixup<<<(a.B + 127) / 128, 128, 0, st>>>(a);
      return cuda_check(cudaGetLastError(), "k_line_dc_fixup");
    }
  }
  return set_error(FSM_ERR_UNSUPPORTED, "1D: unsupported nonlinear term");
}

}  // namespace fsm
